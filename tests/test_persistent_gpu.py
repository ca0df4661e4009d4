"""The persistent kernel where batches that fit on chip no longer reach it:
many programs beside one of 15 qubits, finish times, and device sampling
above 14 qubits in every FP32 form."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _world():
    p2.world_ensure()
    form = p2.get_fp32_form()
    yield
    p2.set_precision(p2.PREC_FP64)
    p2.set_fp32_form(form)
    p2.set_batch_persistent(True)
    p2.set_device_sampling(p2.DEVICE_SAMPLING_AUTO)


def _problems(widths):
    return [dict(nqb=n, terms=workloads.jw_terms(n, 6 + k % 37, seed=k),
                 dets=workloads.hamming_dets(n, 1, max(1, n // 2), seed=k),
                 steps=1 + k % 3, delta=0.11)
            for k, n in enumerate(widths)]


# more programs than lanes, and ten looks of 32, with a wide one among them
MANY = [15] + [5 + k % 8 for k in range(44)]
TINY = [4 + k % 6 for k in range(299)] + [15]


@pytest.mark.parametrize("widths", [MANY, TINY], ids=["45", "300"])
def test_many_programs_fp64(widths, oracle_lib):
    probs = _problems(widths)
    zs, stats = p2.batch("trott2", probs, with_stats=True)
    assert sum(s["launches"] for s in stats) == 1
    assert all(s["finish_ms"] is not None and s["finish_ms"] >= 0
               for s in stats)
    for p, z in zip(probs, zs):
        t, d = p["terms"], p["dets"]
        assert np.array_equal(z, oracle_lib.trott(
            p["nqb"], t.flip, t.phase, t.cf, d.idx, d.cf, p["steps"], 0.11,
            order2=True))


@pytest.mark.parametrize("form", [p2.FORM_LIFTED, p2.FORM_LIFTED_F32,
                                  p2.FORM_LIFTED_MIXED])
def test_many_programs_fp32(form):
    probs = _problems(MANY)
    p2.set_precision(p2.PREC_FP32)
    p2.set_fp32_form(form)
    got = p2.batch("trott", probs)
    p2.set_batch_persistent(False)
    for a, b in zip(got, p2.batch("trott", probs)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", [p2.PREC_FP32, p2.PREC_FP64])
def test_finish_times(prec):
    p2.set_precision(prec)
    probs = _problems([15, 15, 15])
    for p, steps in zip(probs, (2, 2, 40)):
        p["terms"] = workloads.jw_terms(15, 300, seed=steps)
        p["steps"] = steps
    _, stats = p2.batch("trott", probs, with_stats=True)
    fin = [s["finish_ms"] for s in stats]
    assert all(f is not None and f > 0 for f in fin), fin
    assert fin[2] > max(fin[0], fin[1]), fin


@pytest.mark.parametrize("kind", ["qdrift", "cmpsit"])
@pytest.mark.parametrize("form", [p2.FORM_LIFTED, p2.FORM_LIFTED_F32])
def test_device_sampling(form, kind):
    n = 15
    t = workloads.jw_terms(n, 300, seed=0xF64A)
    d = workloads.hamming_dets(n, 3, 7, seed=0xF64B)
    p2.set_precision(p2.PREC_FP32)
    p2.set_fp32_form(form)
    out = []
    for mode in (p2.DEVICE_SAMPLING_OFF, p2.DEVICE_SAMPLING_ON):
        p2.set_device_sampling(mode)
        if kind == "qdrift":
            z, st = p2.qdrift(n, t, d, 5, 200, 0.02, 0x5EE1,
                              with_stats=True, with_state=True)
        else:
            z, st = p2.cmpsit(n, t, d, 3, 2, 40, 90, 0.05, 0.004, 0xC0DF,
                              with_stats=True, with_state=True)
        out.append((z, st))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1]["state"], out[1][1]["state"])
    assert out[1][1]["launches"] < out[0][1]["launches"]
