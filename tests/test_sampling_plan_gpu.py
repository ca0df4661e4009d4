"""The device planner of device sampling under every span and cap: FP32
overlaps depend on where passes end (one rounding each), so equal bits on
the host loop and on the device mean equal plans."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strings", ["jw", "random", "diagonal"])
@pytest.mark.parametrize("fusion", [(1, 0), (2, 3), (3, 0), (4, 1), (5, 0),
                                    (5, 7)])
@pytest.mark.parametrize("n", [4, 9, 15])
def test_device_plan_equals_host_plan(n, fusion, strings):
    make = workloads.jw_terms if strings == "jw" else workloads.random_terms
    t = make(n, 60, seed=10 * n + fusion[0])
    if strings == "diagonal":
        t.flip[5:] = 0
    d = workloads.hamming_dets(n, 2, n // 2, seed=n)
    out = []
    p2.set_precision(p2.PREC_FP32)
    p2.set_fusion(*fusion)
    try:
        for mode in (False, True):
            p2.set_device_sampling(mode)
            z, st = p2.qdrift(n, t, d, 3, 400, 0.05, 0x5EED + n,
                              with_stats=True, with_state=True)
            out.append((z, st["state"], st["passes"]))
    finally:
        p2.set_device_sampling(p2.DEVICE_SAMPLING_AUTO)
        p2.set_fusion(5, 0)
        p2.set_precision(p2.PREC_FP64)
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]
