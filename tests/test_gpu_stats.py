"""fgt_stats against what ran: the launch count against the kernels that the
profiler saw.  Whole numbers: no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTERS = ("k_count_points",)  # kernels of the statistics themselves


def _kernels(f):
    """Result of f() and the names of this library's kernels that it ran."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as pr:
        r = f()
        torch.cuda.synchronize()
    names = [e.name for e in pr.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    return r, [n for n in names if "fgt::" in n and not any(c in n for c in COUNTERS)]


def _case(dim, n, nt, delta, eps, nd=1, pgh=1, dip=False, period=0, **kw):
    rng = np.random.default_rng(3)
    c = dict(nd=nd, dim=dim, delta=delta, eps=eps, iperiod=period, ifpgh=pgh, stats=True,
             sources=rng.uniform(-0.5, 0.5, (n, dim)), charge=rng.standard_normal((n, nd)), **kw)
    if nt:
        c.update(targets=rng.uniform(-0.5, 0.5, (nt, dim)), ifpghtarg=pgh)
    if dip:
        c.update(dipstr=rng.standard_normal((n, nd)), rnormal=rng.standard_normal((n, dim)))
    return c


CASES = {
    "3d_mixed_small": _case(3, 3001, 0, 1e-3, 1e-6),
    "3d_mixed_split_sets": _case(3, 300001, 30001, 1e-3, 1e-3, pgh=2),  # two launches of inverses
    "3d_fp64": _case(3, 9001, 500, 4e-3, 1e-9, pgh=2),
    "3d_fp64_hess": _case(3, 9001, 0, 4e-3, 1e-9, pgh=3, dip=True, nd=2),
    "3d_periodic": _case(3, 9001, 0, 4e-3, 1e-6, period=1),
    "2d_fp64_nd5": _case(2, 20001, 900, 1e-4, 1e-9, nd=5, pgh=2),
    "2d_mixed": _case(2, 20001, 0, 1e-4, 1e-6, pgh=3),
    "1d_deep": _case(1, 5001, 100, 1e-9, 1e-6, ndiv=3),
    "root_only": _case(3, 100, 0, 1e-1, 1e-6),
}


@pytest.mark.parametrize("tree", ["dense", "sorted"])
@pytest.mark.parametrize("name", CASES)
def test_launch_count(fgt, monkeypatch, name, tree):
    if tree == "sorted":
        monkeypatch.setenv("FGT_TREE_SORTED", "1")
    fgt.pfgt(**CASES[name])
    r, names = _kernels(lambda: fgt.pfgt(**CASES[name]))
    assert names, "the profiler saw no kernel"
    assert r["stats"]["n_kernel_launches"] == len(names)
