"""FP64 3D calls on both sides of what the matrix kernels take, against the
oracle's exact plane-wave sums: periodic boxes of 1.1 and 1.9 cut-offs (K above
31 takes the general kernels) and kernel width 16 (the form alone takes them).

Tolerance: the NUFFT's 0.3 eps, as in test_gpu_pw64.py."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


def _check(fgt, oracle, kw):
    ro = oracle.pfgt(**kw)
    out = []
    for small_eval in (-1, 0):
        r = fgt.pfgt(precision=fgt.PREC_FP64, small_eval=small_eval, stats=True, **kw)
        assert r["stats"]["n_form_boxes"] > 0
        for f in ("pot", "grad", "pottarg", "gradtarg"):
            if f in ro:
                assert relerr(ro[f], r[f]) <= 0.3 * kw["eps"], (f, relerr(ro[f], r[f]))
        out.append(r["stats"])
    return out[0]


@pytest.mark.parametrize("eps,ratio", [(1e-9, 1.1), (1e-9, 1.9), (1e-12, 1.1), (1e-12, 1.9)])
def test_periodic_boxes(fgt, oracle, eps, ratio):
    rng = np.random.default_rng(17)
    side = 0.25
    delta = (side / ratio) ** 2 / np.log(1 / eps)
    # full boxes that touch across the border, and a background
    groups = [c + rng.uniform(0.01, 0.24, (300, 3)) for c in
              ([-0.5, -0.5, 0.25], [0.25, -0.5, 0.25], [-0.5, -0.25, -0.5], [0.0, 0.0, 0.0])]
    src = np.concatenate(groups + [rng.uniform(-0.5, 0.5, (200, 3))])
    trg = rng.uniform(-0.5, 0.5, (300, 3))
    st = _check(fgt, oracle, dict(nd=1, dim=3, delta=delta, eps=eps, iperiod=1, bs0=1.0,
                                  cen0=[0.0] * 3, sources=src, ifpgh=2, targets=trg, ifpghtarg=2,
                                  charge=rng.standard_normal((src.shape[0], 1))))
    assert (st["npw"] // 2 > 31) == (ratio > 1.5)


@pytest.mark.parametrize("pgh", [1, 2])
def test_width_16(fgt, oracle, pgh):
    rng = np.random.default_rng(18)
    src = np.concatenate([rng.uniform(-0.4, 0.4, 3) + rng.uniform(-0.03, 0.03, (n, 3))
                          for n in (300, 700)] + [rng.uniform(-0.5, 0.5, (400, 3))])
    st = _check(fgt, oracle, dict(nd=1, dim=3, delta=2e-3, eps=1e-13, iperiod=0, sources=src,
                                  ifpgh=pgh, charge=rng.standard_normal((src.shape[0], 1))))
    assert st["spread_width"] == 16
