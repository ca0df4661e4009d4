"""A device reset between two uses of the library: kernels are configured
again in the new context, and nothing of destroyed registers is reused.
In a child process, whose context the reset ends; registers are destroyed
before it, one of them by a thread that made no other CUDA call."""

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, glob, threading
import numpy as np, torch
import phase2_b200 as p2
from phase2_b200 import Register, workloads

def register(n, prec):
    rng = np.random.Generator(np.random.PCG64(n))
    flip = rng.integers(0, 1 << n, 60).astype(np.uint64)
    phase = rng.integers(0, 1 << n, 60).astype(np.uint64)
    with Register(n, prec) as r:
        r.setamps([3], [1.0])
        r.paulirot(flip, phase, rng.uniform(-1, 1, 60))
        return r.get_state()

def everything():
    out = [register(n, prec) for prec in (p2.PREC_FP64, p2.PREC_FP32)
           for n in (9, 13, 14, 17, 20, 24)]
    for prec in (p2.PREC_FP64, p2.PREC_FP32):
        p2.set_precision(prec)
        for n in (10, 13, 14, 15):
            t = workloads.jw_terms(n, 80, seed=n)
            d = workloads.hamming_dets(n, 1, n // 2, seed=n)
            out.append(p2.qdrift(n, t, d, 16, 40, 0.05, 9))
            out += p2.batch("trott", [dict(nqb=n, terms=t, dets=d, steps=2,
                                           delta=0.1)] * 3)
    out.append(norm())
    th = threading.Thread(target=lambda: register(8, p2.PREC_FP64))
    th.start()
    th.join()
    return out

def norm():
    # phase2_norm2_noalloc on a state of the process's own
    st, res = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(st), 16 << 10) == 0
    assert rt.cudaMalloc(ctypes.byref(res), 16) == 0
    host = np.arange(2 << 10, dtype=np.float64)
    got = np.zeros(2)
    assert rt.cudaMemcpy(st, host.ctypes.data_as(ctypes.c_void_p),
                         ctypes.c_size_t(16 << 10), 1) == 0
    fn = p2.lib().phase2_norm2_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64,
                   ctypes.c_void_p, ctypes.c_void_p]
    assert fn(st, p2.PREC_FP64, 1 << 10, res, None) == 0
    assert rt.cudaMemcpy(got.ctypes.data_as(ctypes.c_void_p), res,
                         ctypes.c_size_t(16), 2) == 0
    assert rt.cudaFree(st) == 0 and rt.cudaFree(res) == 0
    return got

names = glob.glob(torch.__path__[0] + "/../nvidia/cuda_runtime/lib/"
                  "libcudart.so*") + ["libcudart.so.12"]
rt = ctypes.CDLL(names[0])
p2.world_ensure()
want = everything()
assert want[-1][0] == sum(k * k for k in range(2 << 10))
for _ in range(2):
    assert rt.cudaDeviceReset() == 0
    for a, b in zip(want, everything()):
        assert np.array_equal(a, b)
print("same")
"""


def test_reset_between_uses():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
