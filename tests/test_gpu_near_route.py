"""Which near field a call takes, from its FGT_LOG line: packed records in both
precisions, the list walk where FGT_NEAR_PACK_MAX forbids them, where they have
no room (FGT_WORKSPACE_MAX) and for dipoles.  Whole numbers: no tolerance."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CALL = r"""
import numpy as np, fgt_b200 as F
rng = np.random.default_rng(5)
n = 400000
src, q = rng.uniform(-0.5, 0.5, (n, 3)), rng.standard_normal((n, 1))
kw = dict(nd=1, dim=3, delta=4.5e-5, eps=1e-9, iperiod=0, sources=src, ndiv=60, ifpgh=2)
for prec in (F.PREC_FP64, F.PREC_MIXED):
    F.pfgt(charge=q, precision=prec, **kw)
F.pfgt(dipstr=q, rnormal=src, precision=F.PREC_FP64, **kw)
"""


def _records(**env):
    e = dict(os.environ, FGT_LOG="1", **env)
    r = subprocess.run([sys.executable, "-c", CALL], cwd=ROOT, env=e, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return [json.loads(l)["near_records"] for l in r.stderr.splitlines() if l.startswith('{"fgt"')]


def test_near_field_route():
    f64, mixed, dip = _records()
    assert f64 == mixed and f64 * 32 > 200 << 20 and dip == 0  # some 20 records a point
    assert _records(FGT_NEAR_PACK_MAX="0") == [0, 0, 0]
    assert _records(FGT_WORKSPACE_MAX=str(256 << 20)) == [0, 0, 0]
