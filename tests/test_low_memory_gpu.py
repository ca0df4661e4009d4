"""Little free device memory, in a child process that holds the rest: device
sampling falls back on the kernel that needs less scratch, with the same
bits, a flush without room for its plan runs on the pass kernels, and a call
that fails leaves other registers alone."""

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

HEAD = """
import numpy as np, torch
import phase2_b200 as p2
from phase2_b200 import Register, workloads

def leave(mib):
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - (mib << 20), dtype=torch.uint8, device="cuda")

p2.world_ensure()
with Register(20, p2.PREC_FP64) as r:
    r.norm2()
"""

SAMPLING = """
t = workloads.jw_terms(8, 60, seed=1)
d = workloads.hamming_dets(8, 1, 4, seed=2)
def run():
    return p2.qdrift(8, t, d, 3, 1 << 21, 1e-4, 7, with_stats=True,
                     with_state=True)
held = leave(480)
a, sa = run()
del held
torch.cuda.empty_cache()
b, sb = run()
assert np.array_equal(a, b) and np.array_equal(sa["state"], sb["state"])
print("done")
"""

FAILURE = """
held = leave(480)
with Register(17, p2.PREC_FP64) as a, Register(12, p2.PREC_FP64) as b:
    try:
        a.getamps(np.zeros(1 << 25, dtype=np.uint64))
    except RuntimeError:
        b.setamps([5], [2.0])
        b.paulirot(np.array([5], dtype=np.uint64),
                   np.array([0], dtype=np.uint64), np.array([0.0]))
        assert b.norm2() == 4.0
        print("done")
"""

LEAK = """
held = leave(480)
a = Register(17, p2.PREC_FP64)
a.norm2()
before = torch.cuda.mem_get_info()[0]
try:
    a.getamps(np.zeros(1 << 25, dtype=np.uint64))
except RuntimeError:
    a.close()
    assert torch.cuda.mem_get_info()[0] > before - (32 << 20)
    print("done")
"""

CREATION = """
with Register(20, p2.PREC_FP64) as a:
    held = leave(8)
    made = []
    try:
        while True:
            made.append(Register(14, p2.PREC_FP64))
    except RuntimeError:
        a.setamps([5], [2.0])
        a.paulirot(np.array([5], dtype=np.uint64),
                   np.array([0], dtype=np.uint64), np.array([0.0]))
        assert a.norm2() == 4.0
        print("done")
    for r in made:
        r.close()
"""


PLAN = """
n, k = 21, 6000
rng = np.random.Generator(np.random.PCG64(1))
ops = (rng.integers(0, 1 << n, k).astype(np.uint64),
       rng.integers(0, 1 << n, k).astype(np.uint64), rng.uniform(-1, 1, k))
amp = np.zeros(1 << n, dtype=complex)
amp[5] = 1.0
with Register(n, p2.PREC_FP64) as r, Register(n, p2.PREC_FP64) as first:
    # both kinds of kernel and the records' buffer, while there is room
    first.set_state(amp)
    first.paulirot(*ops)
    want = first.get_state()
    p2.lib().phase2_set_fp32_form(p2.FORM_LIFTED_F32)
    with Register(n, p2.PREC_FP32) as f:
        f.paulirot(*ops)
        f.synchronize()
    r.set_fusion(4, 0)
    r.set_state(amp)
    r.paulirot(*ops)
    r.get_state()
    r.set_fusion(5, 0)
    r.set_state(amp)
    # destroyed registers' streams and buffers for those made below
    kept = [Register(10, p2.PREC_FP64) for _ in range(31)]
    for x in kept:
        x.close()
    held = leave(8)
    # then what the pool still has
    rest, m = [], 22
    while m >= 10 and len(rest) < 31:
        try:
            rest.append(Register(m, p2.PREC_FP64))
        except RuntimeError:
            m -= 1
    r.paulirot(*ops)
    assert np.array_equal(r.get_state(), want)
    assert r.stats()["rotations"] == 2 * k
    print("done")
    for x in rest:
        x.close()
"""


def _child(code):
    r = subprocess.run([sys.executable, "-c", HEAD + code], cwd=ROOT,
                       timeout=600, capture_output=True, text=True)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr


def test_device_sampling_without_room_for_sub_passes():
    _child(SAMPLING)


def test_flush_without_room_for_its_plan():
    _child(PLAN)


def test_failed_register_keeps_nothing():
    _child(LEAK)


def test_failure_stays_with_its_register():
    _child(FAILURE)


def test_failed_creation_leaves_others_alone():
    _child(CREATION)
