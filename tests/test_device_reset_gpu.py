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
    th = threading.Thread(target=lambda: register(8, p2.PREC_FP64))
    th.start()
    th.join()
    return out

p2.world_ensure()
want = everything()
names = glob.glob(torch.__path__[0] + "/../nvidia/cuda_runtime/lib/"
                  "libcudart.so*") + ["libcudart.so.12"]
for _ in range(2):
    assert ctypes.CDLL(names[0]).cudaDeviceReset() == 0
    for a, b in zip(want, everything()):
        assert np.array_equal(a, b)
print("same")
"""


def test_reset_between_uses():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
