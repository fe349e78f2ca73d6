"""FP64 3D gradients at six digits, where the evaluation takes the reference
cell's derivative terms (a few 1e-8 of the gradient) out again from sums that
every unit of points leaves in shared memory: many units per warp, handed out in
another order and made up of other points from run to run.

Tolerance: the runs differ by the order of FP64 sums, 1e-13 as in
test_gpu_pw64.py; another unit's sums would show at 1e-8."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


def test_units_keep_their_own_sums(fgt):
    rng = np.random.default_rng(14)
    n = 150001
    src = rng.uniform(-0.5, 0.5, (n, 3))
    kw = dict(nd=1, dim=3, delta=2e-2, eps=1e-6, iperiod=0, sources=src, ifpgh=2, small_eval=0,
              charge=rng.standard_normal((n, 1)), precision=fgt.PREC_FP64, stats=True)
    a = fgt.pfgt(**kw)
    assert a["stats"]["pts_eval_nufft"] == n and a["stats"]["slabs_eval"] == 1
    for _ in range(3):
        b = fgt.pfgt(**kw)
        d = np.abs(b["grad"] - a["grad"]).max() / np.abs(a["grad"]).max()
        assert d < 1e-13 and relerr(a["pot"], b["pot"]) < 1e-13, d
