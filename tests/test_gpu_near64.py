"""FP64 near field on packed records and on the list walk (FGT_NEAR_PACK_MAX=0)
against the exact sums, with items of 1 to 33 points (lane groups of 4, 8, 16
and 32) and record counts around the batch of 32.

Tolerance: with every pair in the near field only terms below eps times the
peak are left out, at most the source count of them; eps = 1e-13 and 2,000
sources give 2e-10 of the peak 1, against sums of order sqrt(n) >= 1 per
point.  The two routes differ by the order of the sums: 1e-13."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("pgh", [1, 2])
def test_fp64_near_field_matches_exact_sums(fgt, oracle, monkeypatch, dim, pgh):
    rng = np.random.default_rng(40 + dim)
    groups = []
    for n in (1, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 64, 65):
        groups.append(rng.uniform(-0.5, 0.5, dim) + rng.uniform(-1e-3, 1e-3, (n, dim)))
    src = np.concatenate(groups + [rng.uniform(-0.5, 0.5, (1000, dim))])
    trg = np.concatenate(groups[::-1])[:, :] + 1e-4
    q = rng.uniform(0.5, 1.0, (src.shape[0], 1))
    kw = dict(nd=1, dim=dim, delta=1e-4, eps=1e-13, iperiod=0, sources=src, charge=q, ifpgh=pgh,
              targets=trg, ifpghtarg=pgh, ndiv=5000, stats=True)
    a = fgt.pfgt(**kw)
    assert a["stats"]["near_pairs"] > 0 and a["stats"]["n_form_boxes"] == 0
    monkeypatch.setenv("FGT_NEAR_PACK_MAX", "0")
    b = fgt.pfgt(**kw)
    ex = oracle.direct_exact(1, dim, 1e-4, src, np.concatenate([src, trg]), charge=q, ifpgh=pgh)
    n = src.shape[0]
    for f, g in (("pot", "pottarg"), ("grad", "gradtarg"))[:pgh]:
        for r in (a, b):
            assert relerr(ex[f][:n], r[f]) < 1e-9
            assert relerr(ex[f][n:], r[g]) < 1e-9
        assert relerr(a[f], b[f]) < 1e-13 and relerr(a[g], b[g]) < 1e-13
