"""world_free gives kept registers and pool memory back, whichever thread
calls it, and registers destroyed after it keep none.  In a child process:
the library's world ends there."""

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import threading
import torch
import phase2_b200 as p2
from phase2_b200 import Register

def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]

p2.world_ensure()
with Register(12, p2.PREC_FP64) as r:
    r.norm2()
before = free()
late = Register(28, p2.PREC_FP64)    # 4 GiB
with Register(28, p2.PREC_FP64):     # kept by the pool
    pass
assert free() < before - (7 << 30)
th = threading.Thread(target=p2.lib().world_free)
th.start()
th.join()
assert before - (5 << 30) < free() < before - (3 << 30)
late.close()
assert free() > before - (64 << 20)
p2.world_ensure()                    # and the world starts again
with Register(12, p2.PREC_FP64) as r:
    r.setamps([0], [1.0])
    assert r.norm2() == 1.0
print("given back")
"""


def test_given_back():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0 and "given back" in r.stdout, r.stdout + r.stderr
