"""Batches that fit on chip: the registers' final states and the composite
driver, against the same problems run one by one (the same bits)."""

import ctypes as C

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _world():
    p2.world_ensure()
    yield
    p2.set_precision(p2.PREC_FP64)


def _batch(kind, problems):
    """p2.batch, with every register read before it is freed."""
    lib, objs, out = p2.lib(), [], []
    try:
        for p in problems:
            obj = p2._KIND[kind][0]()
            hm = p2._hamil(p["nqb"], p["terms"])
            sp_kind, sp_ptr, _keep = p2._initial_state(p["nqb"], p["dets"])
            dt = p2._driver_data(kind, p)
            assert getattr(lib, f"{kind}_init")(
                C.byref(obj), C.byref(dt), hm, sp_kind, sp_ptr, None) == 0
            objs.append(obj)
        arr = (C.c_void_p * len(objs))(
            *[C.cast(C.pointer(o), C.c_void_p) for o in objs])
        assert getattr(lib, f"{kind}_simul_batch")(arr, len(objs)) == 0
        for p, o in zip(problems, objs):
            amp = np.empty(1 << p["nqb"], dtype=np.complex128)
            assert lib.qreg_get_state(
                C.byref(o.ct.reg),
                amp.ctypes.data_as(C.POINTER(C.c_double))) == 0
            out.append((p2._values(o.ct.vals), amp))
    finally:
        for o in objs:
            getattr(lib, f"{kind}_free")(C.byref(o))
    return out


@pytest.mark.parametrize("prec", [p2.PREC_FP64, p2.PREC_FP32])
@pytest.mark.parametrize("kind", ["trott", "qdrift", "cmpsit"])
@pytest.mark.parametrize("widths", [(4, 9, 11), (14, 5, 8, 13),
                                    (12, 7, 3 + 1)])
def test_states(widths, kind, prec):
    p2.set_precision(prec)
    probs = []
    for k, n in enumerate(widths):
        probs.append(dict(
            nqb=n, terms=workloads.jw_terms(n, 20 + 9 * k, seed=k),
            dets=workloads.hamming_dets(n, 1 + k % 2, n // 2, seed=9 + k),
            steps=2, delta=0.1, samples=2, depth=25, step_size=0.05, length=7,
            angle_det=0.05, angle_rand=0.01, seed=3 + k))
    p2.set_device_sampling(p2.DEVICE_SAMPLING_OFF)
    try:
        for p, (z, amp) in zip(probs, _batch(kind, probs)):
            head = (p["nqb"], p["terms"], p["dets"])
            kw = dict(with_stats=True, with_state=True)
            if kind == "trott":
                want, st = p2.trott(*head, 2, 0.1, **kw)
            elif kind == "qdrift":
                want, st = p2.qdrift(*head, 2, 25, 0.05, p["seed"], **kw)
            else:
                want, st = p2.cmpsit(*head, 2, 2, 7, 25, 0.05, 0.01,
                                     p["seed"], **kw)
            assert np.array_equal(z, want)
            assert np.array_equal(amp, st["state"])
    finally:
        p2.set_device_sampling(p2.DEVICE_SAMPLING_AUTO)
