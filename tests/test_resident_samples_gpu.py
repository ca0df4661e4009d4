"""Samples run whole on chip: sample counts on both sides of every block
count, several chunks of the host queue, head terms, repeated and unordered
determinants; overlaps, final register and generator as on the host loop."""

import subprocess
import sys

import numpy as np
import pytest

import phase2_b200 as p2
from conftest import ROOT
from phase2_b200 import Dets, workloads

pytestmark = pytest.mark.gpu


def _both(kind, prec, *args):
    out = []
    p2.set_precision(prec)
    try:
        for mode in (False, True):
            p2.set_device_sampling(mode)
            z, st = getattr(p2, kind)(*args, with_stats=True,
                                      with_state=True)
            out.append((z, st["state"], st["passes"]))
    finally:
        p2.set_device_sampling(p2.DEVICE_SAMPLING_AUTO)
        p2.set_precision(p2.PREC_FP64)
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", [p2.PREC_FP64, p2.PREC_FP32])
@pytest.mark.parametrize("n,samples,depth", [
    (4, 1, 5), (10, 90, 40), (11, 3, 9000), (12, 1, 70), (12, 80, 60),
    (13, 9, 60), (13, 20, 60), (13, 75, 20), (14, 2, 60), (14, 20, 60), (14, 40, 60),
    (14, 80, 20)])
def test_qdrift(n, samples, depth, prec):
    t = workloads.jw_terms(n, 50, seed=n + samples)
    # a determinant written twice: the later value holds
    idx = np.array([3, 1, 3, (1 << n) - 1], dtype=np.uint64)
    d = Dets(idx, np.array([0.1, 0.5j, -0.6, 0.3 + 0.2j]))
    _both("qdrift", prec, n, t, d, samples, depth, 0.05, 77)


@pytest.mark.parametrize("prec", [p2.PREC_FP64, p2.PREC_FP32])
@pytest.mark.parametrize("n,length,depth", [(5, 7, 0), (12, 30, 20),
                                            (14, 25, 9)])
def test_cmpsit(n, length, depth, prec):
    t = workloads.jw_terms(n, 60, seed=n)
    d = workloads.hamming_dets(n, 2, n // 2, seed=n)
    _both("cmpsit", prec, n, t, d, 3, 2, length, depth, 0.05, 0.01, 99)


@pytest.mark.parametrize("prec", ["FP64", "FP32"])
@pytest.mark.parametrize("n,samples", [(12, 80), (13, 80), (14, 2)])
def test_first_run_of_a_process(n, samples, prec):
    """A process whose first register is wide: the kernel its sample count
    chooses is configured without any other having run."""
    code = (f"import phase2_b200 as p2\n"
            f"from phase2_b200 import workloads as w\n"
            f"p2.world_ensure(); p2.set_precision(p2.PREC_{prec})\n"
            f"t = w.jw_terms({n}, 50, seed=1)\n"
            f"d = w.hamming_dets({n}, 1, {n} // 2, seed=2)\n"
            f"p2.set_device_sampling(True)\n"
            f"assert len(p2.qdrift({n}, t, d, {samples}, 20, 0.05, 3))"
            f" == {samples}\n")
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT)
