"""Batches whose registers all fit on chip: one launch, every program the
oracle's bits, uneven widths down to registers that do not share out among a
cluster's blocks, all drivers, instances without outputs, and the registers'
final states; a wider register sends the batch to the persistent kernel."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import workloads

pytestmark = pytest.mark.gpu


def _problems(widths, steps):
    out = []
    for k, n in enumerate(widths):
        t = workloads.jw_terms(n, 20 + 17 * k, seed=40 + k)
        d = workloads.hamming_dets(n, 1 + k % 3, n // 2, seed=80 + k)
        out.append(dict(nqb=n, terms=t, dets=d, steps=steps[k % len(steps)],
                        delta=0.1, samples=1 + k % 3, depth=30 + k,
                        step_size=0.05, seed=5 + k))
    return out


@pytest.mark.parametrize("kind", ["trott", "trott2", "qdrift"])
@pytest.mark.parametrize("widths", [
    (4, 9, 11), (14, 5, 8, 14, 13), (12, 12), (13, 4) * 20,
    (14, 10, 15)])
def test_oracle_bits(widths, kind, oracle_lib):
    probs = _problems(widths, (3, 1, 2) if kind != "qdrift" else (1,))
    zs, stats = p2.batch(kind, probs, with_stats=True)
    assert sum(s["launches"] for s in stats) == 1
    assert all(s["finish_ms"] > 0 for s in stats)
    for p, z in zip(probs, zs):
        t, d = p["terms"], p["dets"]
        args = (p["nqb"], t.flip, t.phase, t.cf, d.idx, d.cf)
        if kind == "qdrift":
            want = oracle_lib.qdrift(*args, p["samples"], p["depth"], 0.05,
                                     p["seed"])
        else:
            want = oracle_lib.trott(*args, p["steps"], 0.1,
                                    order2=kind == "trott2")
        assert np.array_equal(z, want)


def test_no_outputs_beside_others(oracle_lib):
    probs = _problems((6, 13, 12), (2, 0, 1))
    zs = p2.batch("trott", probs)
    assert len(zs[1]) == 0
    for k in (0, 2):
        p, t, d = probs[k], probs[k]["terms"], probs[k]["dets"]
        assert np.array_equal(zs[k], oracle_lib.trott(
            p["nqb"], t.flip, t.phase, t.cf, d.idx, d.cf, p["steps"], 0.1))


def test_fp32_equals_streams():
    probs = _problems((14, 6, 13, 12, 9), (3, 1, 2))
    p2.set_precision(p2.PREC_FP32)
    try:
        got = p2.batch("trott2", probs)
        p2.set_batch_persistent(False)
        want = p2.batch("trott2", probs)
    finally:
        p2.set_batch_persistent(True)
        p2.set_precision(p2.PREC_FP64)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
