"""ttfld_sor_solve_noalloc runs on the stream it is given and on no other: its
first call in a process, without a context, returns while another stream of the
caller's (one that the legacy default stream waits for) is still busy.

The other stream is held by a host function that waits for the call's return,
20 s at most; so a call that waits for that stream too returns after it.  In a
process of its own, for the first call, with every kernel loaded beforehand."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = r"""
import ctypes, os, sys, threading
import numpy as np
from ttcode_gb300 import _ffi

try:
    rt = ctypes.CDLL("libcudart.so")
except OSError:
    rt = ctypes.CDLL(os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "lib64", "libcudart.so"))
L = _ffi.lib()
vp = ctypes.c_void_p

def ok(rc):
    assert rc == 0, rc

def device(a):
    p = vp()
    ok(rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(a.nbytes)))
    ok(rt.cudaMemcpy(p, vp(a.ctypes.data), ctypes.c_size_t(a.nbytes), 1))
    return p

nx, ny, nz = 24, 16, 12
ok(rt.cudaSetDevice(0))
cells = [np.full((nz, ny, nx), v) for v in (7.0, -1.0, -1.0, -1.0, -1.0, -1.0, -1.0, 1.0)]
ptrs = [device(a) for a in cells]
x = np.zeros((nz + 4, ny + 4, nx + 4))
px = device(x)
busy, mine = vp(), vp()
ok(rt.cudaStreamCreate(ctypes.byref(busy)))
ok(rt.cudaStreamCreateWithFlags(ctypes.byref(mine), 1))
returned, over = threading.Event(), threading.Event()

@ctypes.CFUNCTYPE(None, vp)
def hold(_):
    returned.wait(20.0)
    over.set()

ok(rt.cudaLaunchHostFunc(busy, hold, None))
it = ctypes.c_int()
rc = L.ttfld_sor_solve_noalloc(*ptrs, px, nx, ny, nz, 1.2, 1e-8, 1, 1000, mine, ctypes.byref(it), None, None)
waited = over.is_set()
returned.set()
ok(rt.cudaStreamSynchronize(busy))
assert rc == 0 and it.value > 1, (rc, it.value)
assert not waited, "the call waited for another stream"
print("did not wait")
"""


def test_first_call_waits_for_its_own_stream_only():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, CUDA_MODULE_LOADING="EAGER", PYTHONPATH=ROOT))
    assert r.returncode == 0 and "did not wait" in r.stdout, r.stdout + r.stderr
