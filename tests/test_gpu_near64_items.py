"""FP64 near field on packed records with many items per warp: 32,768 isolated
groups of 17 to 32 points, so an item is one batch of records on all 32 lanes
and its staging buffer is the next item's too.

Tolerance: every pair of a group is within the cut-off; the terms between
groups (0.03 apart, 91 delta) are below 1e-39.  Sums of at most 32 terms of
one sign in another order differ by at most 32 roundings, 4e-15 of the sum; a
coordinate difference of about 3e-4 carries the rounding of two offsets below
0.016, 4e-18 or 1.3e-14 of it: 1e-13 holds both."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


def test_items_of_one_batch(fgt):
    rng = np.random.default_rng(9)
    g = 32
    cen = np.stack(np.meshgrid(*[(np.arange(g) + 0.5) / g - 0.5] * 3, indexing="ij"), -1).reshape(-1, 3)
    ncl = len(cen)
    size = rng.integers(17, 33, ncl)
    delta = 1e-5
    pts = cen[:, None, :] + rng.uniform(-1, 1, (ncl, 32, 3)) * 5e-4
    q = rng.uniform(0.5, 1.0, (ncl, 32))
    live = np.arange(32)[None, :] < size[:, None]
    d = pts[:, :, None, :] - pts[:, None, :, :]
    e = np.exp(-(d * d).sum(-1) / delta) * (q * live)[:, None, :]
    pot = e.sum(-1)
    grad = (-2.0 / delta) * np.einsum("cij,cijk->cik", e, d)
    order = rng.permutation(int(live.sum()))  # no run of a group in input order
    src, qs = pts[live][order], q[live][order][:, None]
    r = fgt.pfgt(nd=1, dim=3, delta=delta, eps=1e-13, iperiod=0, sources=src, charge=qs, ifpgh=2,
                 ndiv=32, precision=fgt.PREC_FP64, stats=True)
    assert r["stats"]["near_pairs"] > 0 and r["stats"]["n_form_boxes"] == 0
    assert relerr(pot[live][order], r["pot"]) < 1e-13
    assert relerr(grad[live][order], r["grad"]) < 1e-13
