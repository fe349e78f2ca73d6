"""Device memory of FP64 3D calls: what the plane-wave grids add to a thread's
workspace, and calls whose workspace has no room for what they would like
(FGT_WORKSPACE_MAX, bytes).  Children of their own, since a thread's workspace
stays with it.

Tolerance: the same sums but for the order of the FP64 atomics (1e-13 in
test_gpu_pw64.py; the groups here are ten times as large: 1e-12)."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

HEAD = r"""
import json, os, sys, threading
import numpy as np, torch
import fgt_b200 as F
rng = np.random.default_rng(21)
def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(a))
def call(**kw):
    return F.pfgt(precision=F.PREC_FP64, **kw)
def in_thread(env, **kw):
    '''result, and the device memory that the call's thread holds after it'''
    os.environ.update(env)
    out = []
    def go():
        torch.cuda.init()
        f0 = torch.cuda.mem_get_info()[0]
        try:
            for _ in range(2):  # the second in one consolidated chunk
                r = call(**kw)
            out.append((r, f0 - torch.cuda.mem_get_info()[0]))
        except F.FgtError as e:
            out.append((None, e.code))
    t = threading.Thread(target=go); t.start(); t.join()
    for k in env: del os.environ[k]
    return out[0]
"""


def _child(code):
    r = subprocess.run([sys.executable, "-c", HEAD + code], cwd=ROOT, capture_output=True,
                       text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr[-3000:]
    return json.loads(r.stdout.splitlines()[-1])


GRIDS = r"""
n = 300000
src = rng.uniform(-0.5, 0.5, (n, 3))
q = rng.standard_normal((n, 1))
kw = dict(nd=1, dim=3, delta=1.5e-4, eps=1e-9, iperiod=0, sources=src, charge=q, ifpgh=2,
          ndiv=30, small_eval=0, stats=True)
call(**kw)  # modules
few, held_few = in_thread({"FGT_GRID64_BOXES": "1"}, **kw)
all_, held = in_thread({}, **kw)
tight, _ = in_thread({"FGT_WORKSPACE_MAX": str(held_few + (300 << 20))}, **kw)
st = all_["stats"]
print(json.dumps(dict(few=held_few, held=held, boxes=[st["n_form_boxes"], st["n_eval_boxes"]],
                      total=torch.cuda.mem_get_info()[1], tight_ok=tight is not None,
                      err=[max(rel(all_[f], r[f]) for f in ("pot", "grad"))
                           for r in (few, tight) if r is not None])))
"""


def test_fp64_grids_hold_a_bounded_share_of_the_device():
    d = _child(GRIDS)
    # boxes enough that all their grids (560 kB each) are far above the bound
    assert min(d["boxes"]) * 560e3 > 2 * d["total"] / 128, d
    # one buffer for the form and the evaluation, kept with 5% of room
    assert d["held"] - d["few"] <= 1.1 * d["total"] / 128, d
    assert d["tight_ok"], d  # fewer grids where there is room for 300 MB of them
    assert max(d["err"]) < 1e-12, d


RECORDS = r"""
n = 400000
src = rng.uniform(-0.5, 0.5, (n, 3))
q = rng.standard_normal((n, 1))
# boxes of about 12 points and the size of the cut-off: some 20 records a point
kw = dict(nd=1, dim=3, delta=4.5e-5, eps=1e-9, iperiod=0, sources=src, charge=q, ifpgh=2,
          ndiv=60, stats=True)
a, held = in_thread({}, **kw)
b, code = in_thread({"FGT_WORKSPACE_MAX": str(256 << 20)}, **kw)
print(json.dumps(dict(held=held, form=a["stats"]["n_form_boxes"], ok=b is not None, code=code,
                      err=[rel(a[f], b[f]) for f in ("pot", "grad")] if b else None)))
"""


def test_fp64_near_field_without_room_for_its_records():
    d = _child(RECORDS)
    assert d["form"] == 0 and d["held"] > 300 << 20, d  # more than the second call may have
    assert d["ok"], d
    assert max(d["err"]) < 1e-12, d
