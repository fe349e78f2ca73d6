"""fgt_stats against what ran: the launch count against the kernels that the
profiler saw, the translation's bytes against the lists of the debug tree; and
no group tables in calls that translate by lists.  Whole numbers: no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTERS = ("k_count_points", "k_count_sources")  # kernels of the statistics themselves


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


# ndiv below the points of a box of the cut-off's size: plane waves in all but the last two
CASES = {
    "3d_mixed_small": _case(3, 3001, 0, 1e-3, 1e-6, ndiv=2),
    "3d_mixed_split_sets": _case(3, 300001, 30001, 1e-3, 1e-3, pgh=2, ndiv=20),  # two launches of inverses
    "3d_fp64": _case(3, 9001, 500, 4e-3, 1e-9, pgh=2, ndiv=20),
    "3d_fp64_hess": _case(3, 9001, 0, 4e-3, 1e-9, pgh=3, dip=True, nd=2, ndiv=20),
    "3d_periodic": _case(3, 9001, 0, 4e-3, 1e-6, period=1, ndiv=20),
    "2d_fp64_nd5": _case(2, 20001, 900, 1e-4, 1e-9, nd=5, pgh=2, ndiv=10),
    "2d_mixed": _case(2, 20001, 0, 1e-4, 1e-6, pgh=3, ndiv=10),
    "1d": _case(1, 5001, 100, 1e-6, 1e-6, ndiv=3),
    "1d_deep": _case(1, 5001, 100, 1e-12, 1e-6),
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
    assert (r["stats"]["n_form_boxes"] > 0) == (name not in ("1d_deep", "root_only"))
    assert r["stats"]["n_kernel_launches"] == len(names)


@pytest.mark.parametrize("dim,delta,nd,prec", [
    (1, 1e-4, 1, "fp64"), (1, 1e-4, 1, "mixed"), (2, 1e-3, 2, "fp64"), (2, 1e-3, 1, "mixed"),
    (3, 4e-3, 1, "fp64"), (3, 4e-3, 2, "mixed"),
])
def test_translation_bytes(fgt, dim, delta, nd, prec):
    """By groups (1D, 2D, FP64) the children of one parent read every expansion
    around them once; by lists every box reads its own and its list's."""
    rng = np.random.default_rng(8)
    n = {1: 3000, 2: 9000, 3: 20000}[dim]
    src = rng.uniform(-0.5, 0.5, (n, dim)) ** 3 * 4  # dense in the middle: some boxes are leaves
    fp64 = prec == "fp64"
    st = fgt.pfgt(nd, dim, delta, 1e-6, 0, src, charge=rng.standard_normal((n, nd)), stats=True,
                  precision=fgt.PREC_FP64 if fp64 else fgt.PREC_MIXED)["stats"]
    t = fgt.debug_tree(dim, delta, 1e-6, 0, src, None)
    ptr, lst, own = t["trans_ptr"], t["trans_src"], t["eval_self"]
    assert t["n_trans"] > 0 and t["n_form"] < t["n_eval"]
    if dim < 3 or fp64:
        sets = {}
        for e, b in enumerate(t["eval_box"]):
            s = sets.setdefault(t["parent"][b], set())
            s.update(lst[ptr[e]:ptr[e + 1]])
            s.update([own[e]] if own[e] >= 0 else [])
        reads = sum(len(s) for s in sets.values())
    else:
        reads = t["n_trans"] + t["n_eval"]
    nexp = (st["npw"] + 1) ** (dim - 1) * (st["npw"] // 2 + 1)  # modes -npw/2 .. npw/2, half of one
    assert st["bytes_translate"] == (16 if fp64 else 8) * nexp * nd * (reads + t["n_eval"])


@pytest.mark.parametrize("name", ["3d_mixed_split_sets", "3d_periodic", "3d_fp64", "2d_mixed"])
def test_groups_only_where_they_are_read(fgt, name):
    fgt.pfgt(**CASES[name])
    _, names = _kernels(lambda: fgt.pfgt(**CASES[name]))
    assert any("k_translate" in n for n in names)
    assert any("k_groups" in n for n in names) == any("k_translate_groups" in n for n in names)
