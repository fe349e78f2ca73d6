"""Translation by sibling groups against the oracle: 1D to 3D, both
precisions, several densities, free space and periodic (from the smallest
number of boxes a side), dense and sparse neighbourhoods, groups with
children that hold no targets or no sources.

Tolerance: as in test_gpu_pfgt.py, the NUFFT's 0.3 eps in FP64; the mixed
path adds its FP32 sums, a few 1e-6 of the largest value."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,delta,period,nd", [
    (1, 1e-4, 0, 1), (1, 1e-3, 1, 2),
    (2, 2e-3, 0, 2), (2, 1e-3, 1, 1), (2, 1.2e-2, 1, 1),
    (3, 4e-3, 0, 1), (3, 4e-3, 1, 2), (3, 1.2e-2, 1, 1), (3, 2e-2, 0, 1),
])
@pytest.mark.parametrize("shape", ["dense", "sparse"])
def test_groups_match_oracle(fgt, oracle, dim, delta, period, nd, shape):
    rng = np.random.default_rng(11)
    n = {1: 2000, 2: 6000, 3: 9000}[dim]
    src, trg = rng.uniform(-0.5, 0.5, (2, n, dim))
    if shape == "sparse":  # sources near a diagonal, targets on one side of a plane
        src = np.clip(src[:, :1] + 0.02 * src, -0.499, 0.499)
        trg[:, 0] = -np.abs(trg[:, 0])
    kw = dict(nd=nd, dim=dim, delta=delta, eps=1e-6, iperiod=period, sources=src, bs0=1.0,
              cen0=[0.0] * dim, charge=rng.standard_normal((n, nd)), ifpgh=1, targets=trg,
              ifpghtarg=1)
    ro = oracle.pfgt(**kw)
    for prec, tol in ((fgt.PREC_FP64, 0.3e-6), (fgt.PREC_MIXED, 4e-6)):
        r = fgt.pfgt(precision=prec, stats=True, **kw)
        for f in ("pot", "pottarg"):
            assert relerr(ro[f], r[f]) <= tol, (f, prec, relerr(ro[f], r[f]), r["stats"]["n_form_boxes"])
