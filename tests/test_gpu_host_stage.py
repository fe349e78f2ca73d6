"""Small host-array calls and their pinned staging: after a call that failed
half way on a stream of the caller's, which the caller then destroys, the
thread's next small call gives the results of a call in a fresh thread; and
strengths or outputs that lie in device memory do not end the process.

Tolerance: equal calls differ by the order of FP32 atomics only, as in
test_gpu_failure.py (1e-6)."""
import ctypes as C
import subprocess
import sys
import threading

import numpy as np
import pytest

from conftest import ROOT, relerr

pytestmark = pytest.mark.gpu


def _inputs():
    rng = np.random.default_rng(12)
    src, trg = rng.uniform(-0.5, 0.5, (2, 2000, 3))
    return src, trg, rng.standard_normal((2000, 1))


def _call(fgt, delta, stream=0):
    """pot and pottarg of the status call with host arrays on `stream`."""
    L = fgt.lib()
    src, trg, q = _inputs()
    pot, pt = np.zeros((2, 2000, 1))
    o = fgt.FgtOpts()
    L.fgt_opts_default(C.byref(o))
    o.stream = stream
    b0, c0 = C.c_double(1.0), np.zeros(3)

    def p(a):
        return a.ctypes.data_as(C.c_void_p)

    rc = L.fgt_pfgt_c(C.byref(o), 1, 3, delta, 1e-6, 0, C.byref(b0),
                      c0.ctypes.data_as(C.POINTER(C.c_double)), 2000, p(src), 1, p(q), 0, None,
                      None, 1, p(pot), None, None, 2000, p(trg), 1, p(pt), None, None)
    return rc, pot, pt


def _in_fresh_thread(f):
    out = []
    t = threading.Thread(target=lambda: out.append(f()))
    t.start()
    t.join()
    return out[0]


def test_call_after_a_failed_call_whose_stream_is_gone(fgt):
    import torch
    rt = torch.cuda.cudart()
    rc, pot, pt = _in_fresh_thread(lambda: _call(fgt, 1e-3))
    assert rc == fgt.FGT_OK

    def failed_then_good():
        torch.cuda.init()
        s = C.c_void_p()
        assert int(rt.cudaStreamCreate(C.addressof(s))) == 0
        first = _call(fgt, 1e-16, s.value)[0]  # deeper than the path key holds
        assert int(rt.cudaStreamDestroy(s.value)) == 0
        return first, [_call(fgt, 1e-3) for _ in range(2)]

    first, after = _in_fresh_thread(failed_then_good)
    assert first == fgt.FGT_ERR_UNSUPPORTED
    for rc, a, b in after:
        assert rc == fgt.FGT_OK
        assert relerr(pot, a) < 1e-6 and relerr(pt, b) < 1e-6


def test_device_arrays_among_host_arrays():
    """Host sources, so the call is staged; the charges and the potential in
    device memory.  In a child: a fault there would end the process."""
    code = r"""
import ctypes as C, numpy as np, torch, fgt_b200 as F
rng = np.random.default_rng(12)
n = 2000
src, q = rng.uniform(-0.5, 0.5, (n, 3)), rng.standard_normal((n, 1))
ref = F.pfgt(1, 3, 1e-3, 1e-6, 0, src, charge=q, ifpgh=2)
dq = torch.from_numpy(q).cuda()
pot = torch.zeros(n, 1, dtype=torch.float64, device="cuda")
grad = np.zeros((n, 3, 1))
torch.cuda.synchronize()
b0, c0 = C.c_double(1.0), np.zeros(3)
p = lambda a: a.ctypes.data_as(C.c_void_p)
rc = F.lib().fgt_pfgt_c(None, 1, 3, 1e-3, 1e-6, 0, C.byref(b0),
                        c0.ctypes.data_as(C.POINTER(C.c_double)), n, p(src), 1, dq.data_ptr(), 0,
                        None, None, 2, pot.data_ptr(), p(grad), None, 0, None, 0, None, None, None)
assert rc == F.FGT_OK, F.last_error()
rel = lambda a, b: np.linalg.norm(a - b) / np.linalg.norm(a)
assert rel(ref["pot"], pot.cpu().numpy()) < 1e-6 and rel(ref["grad"], grad) < 1e-6
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
