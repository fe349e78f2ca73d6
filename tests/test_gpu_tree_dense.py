"""The tree over dense cell tables against the tree from sorted keys (the
general path, FGT_TREE_SORTED=1): the same boxes, ranges, point order and
reference boxes for every dimension, depth and point layout that it takes."""
import numpy as np
import pytest

from fgt_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _cases():
    rng = np.random.default_rng(31)
    u = W.uniform
    tight = np.concatenate([u(rng, 5000, 3) * 1e-3 + 0.2, u(rng, 3, 3)])
    line = np.zeros((4001, 3))
    line[:, 0] = np.linspace(-0.5, 0.5, 4001)
    return [
        ("3d_one_point", 3, 1e-3, 0, u(rng, 1, 3), u(rng, 1, 3), 0),
        ("3d_few", 3, 1e-3, 0, u(rng, 40, 3), None, 0),
        ("3d_tight", 3, 1e-5, 0, tight, u(rng, 700, 3), 0),
        ("3d_line", 3, 1e-4, 0, line, None, 7),
        ("3d_root", 3, 1e-1, 0, u(rng, 3000, 3), u(rng, 10, 3), 0),
        ("3d_periodic", 3, 1e-3, 1, u(rng, 9001, 3), None, 20),
        ("2d_clusters", 2, 1e-6, 0, W.gaussian_clusters(rng, 20003, 2, ncl=6), u(rng, 999, 2), 0),
        ("2d_periodic", 2, 1e-5, 1, u(rng, 30001, 2), None, 0),
        ("1d", 1, 1e-7, 0, u(rng, 6001, 1), u(rng, 100, 1), 0),
        ("1d_deep", 1, 1e-12, 0, W.gaussian_clusters(rng, 6001, 1, ncl=3), None, 3),
        ("3d_many_points", 3, 1e-5, 0, W.sphere_surface(rng, 300001), u(rng, 70001, 3), 0),
    ]


@pytest.mark.parametrize("case", _cases(), ids=lambda c: c[0])
def test_dense_tree_equals_sorted_tree(fgt, monkeypatch, case):
    name, dim, delta, iper, src, trg, ndiv = case
    kw = dict(bs0=1.0, cen0=[0.0] * dim, ndiv=ndiv)
    a = fgt.debug_tree(dim, delta, 1e-6, iper, src, trg, **kw)
    monkeypatch.setenv("FGT_TREE_SORTED", "1")
    b = fgt.debug_tree(dim, delta, 1e-6, iper, src, trg, **kw)
    assert a.keys() == b.keys()
    for k in b:
        assert np.array_equal(a[k], b[k]), (name, k)
