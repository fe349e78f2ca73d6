"""FP64 3D form, evaluation and modal sums on the matrix instructions
(fgt_pw64.cu) against the oracle's exact plane-wave sums, at the edges of
their tiles: kernel widths 6-16, blocks with 1, 8, 9, 16, 17, 64, 65 and
more than 8192 points (several sort chunks), several densities, dipoles,
hessians, boxes below the modal threshold, several runs over the boxes.

Tolerance: the FP64 path differs from the oracle by its own NUFFT only,
0.3 eps (as in test_gpu_pfgt.py)."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
FIELDS = ("pot", "grad", "hess", "pottarg", "gradtarg", "hesstarg")


def points(seed, big):
    """Groups of the listed sizes, each inside one grid cell or two, one group
    of `big` points, and a uniform background."""
    rng = np.random.default_rng(seed)
    out = []
    for k, n in enumerate((1, 8, 9, 16, 17, 64, 65, 300, big)):
        c = rng.uniform(-0.45, 0.45, 3)
        out.append(c + rng.uniform(-1e-3, 1e-3, (n, 3)) * (1 if k % 2 else 10))
    out.append(rng.uniform(-0.5, 0.5, (500, 3)))
    return np.concatenate(out)


@pytest.mark.parametrize("eps,pgh,nd,dip,big", [
    (1e-3, 1, 1, False, 400),
    (1e-3, 2, 1, False, 9001),
    (1e-4, 3, 1, True, 400),
    (1e-6, 1, 2, False, 400),
    (1e-6, 2, 1, True, 400),
    (1e-8, 1, 1, False, 400),
    (1e-8, 2, 2, False, 400),
    (1e-9, 2, 1, False, 9001),
    (1e-10, 1, 1, True, 400),
    (1e-10, 3, 1, False, 400),
    (1e-12, 2, 1, True, 400),
])
def test_matrix_kernels_match_oracle(fgt, oracle, eps, pgh, nd, dip, big):
    src, trg = points(1, big), points(2, 70)
    rng = np.random.default_rng(3)
    n = src.shape[0]
    kw = dict(nd=nd, dim=3, delta=4e-3, eps=eps, iperiod=0, sources=src,
              charge=rng.standard_normal((n, nd)), ifpgh=pgh, targets=trg, ifpghtarg=pgh)
    if dip:
        kw.update(dipstr=rng.standard_normal((n, nd)), rnormal=rng.standard_normal((n, 3)))
    ro = oracle.pfgt(**kw)
    for small_eval in (-1, 0):  # modal sums for the small boxes; grids for every box
        r = fgt.pfgt(precision=fgt.PREC_FP64, small_eval=small_eval, stats=True, **kw)
        assert r["stats"]["n_form_boxes"] > 0
        for f in FIELDS:
            if f in ro:
                assert relerr(ro[f], r[f]) <= 0.3 * eps, (f, relerr(ro[f], r[f]))


@pytest.mark.parametrize("eps,pgh,nd,dip,period", [
    (1e-3, 1, 1, False, 0),
    (1e-3, 2, 2, False, 1),
    (1e-6, 2, 1, True, 0),
    (1e-8, 1, 3, False, 0),
    (1e-9, 2, 2, False, 0),
    (1e-10, 1, 1, False, 1),
    (1e-12, 2, 1, True, 0),
    (1e-13, 1, 1, False, 0),
])
def test_2d_matrix_kernels_match_oracle(fgt, oracle, eps, pgh, nd, dip, period):
    """Small 2D boxes: groups of 81 to 2,049 points (the last beyond the
    warp-per-box kernels), counts off the batches of 16 and steps of 4."""
    rng = np.random.default_rng(6)
    groups = [rng.uniform(-0.4, 0.4, 2) + rng.uniform(-5e-3, 5e-3, (n, 2))
              for n in (81, 82, 96, 97, 100, 2048, 2049)]
    src = np.concatenate(groups + [rng.uniform(-0.5, 0.5, (700, 2))])
    trg = rng.uniform(-0.5, 0.5, (333, 2))
    n = src.shape[0]
    kw = dict(nd=nd, dim=2, delta=2e-3, eps=eps, iperiod=period, sources=src, bs0=1.0,
              cen0=[0.0, 0.0], charge=rng.standard_normal((n, nd)), ifpgh=pgh, targets=trg,
              ifpghtarg=pgh)
    if dip:
        kw.update(dipstr=rng.standard_normal((n, nd)), rnormal=rng.standard_normal((n, 2)))
    ro = oracle.pfgt(**kw)
    for small_eval in (-1, 0):
        r = fgt.pfgt(precision=fgt.PREC_FP64, small_eval=small_eval, stats=True, **kw)
        assert r["stats"]["n_form_boxes"] > 0
        for f in FIELDS:
            if f in ro:
                assert relerr(ro[f], r[f]) <= 0.3 * eps, (f, relerr(ro[f], r[f]))


def test_several_runs_over_the_boxes(fgt, monkeypatch):
    """Grids of a few boxes held at a time give the sums of all at once (equal
    but for the order of the atomics)."""
    src = points(4, 2000)
    rng = np.random.default_rng(5)
    kw = dict(nd=1, dim=3, delta=4e-3, eps=1e-9, iperiod=0, sources=src,
              charge=rng.standard_normal((src.shape[0], 1)), ifpgh=2, small_eval=0, ndiv=40)
    a = fgt.pfgt(stats=True, **kw)
    assert a["stats"]["n_eval_boxes"] > 7
    monkeypatch.setenv("FGT_GRID64_BOXES", "3")
    b = fgt.pfgt(**kw)
    for f in ("pot", "grad"):
        assert relerr(a[f], b[f]) < 1e-13
