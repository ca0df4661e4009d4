"""Batches of 14-qubit programs around the counts at which their blocks, or
the kernel, change: the oracle's bits (FP64), the stream mode's (FP32)."""

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
    p2.set_batch_persistent(True)


def _problems(count):
    out = []
    for k in range(count):
        out.append(dict(nqb=14, terms=workloads.jw_terms(14, 24, seed=k % 9),
                        dets=workloads.hamming_dets(14, 1, 7, seed=k % 7),
                        steps=1, delta=0.1, samples=1, depth=16,
                        step_size=0.05, seed=k + 1))
    return out


@pytest.mark.parametrize("kind,count", [
    ("trott", 18), ("trott", 19), ("trott", 32), ("trott", 33),
    ("qdrift", 148), ("qdrift", 149)])
def test_oracle_bits(kind, count, oracle_lib):
    probs = _problems(count)
    zs, stats = p2.batch(kind, probs, with_stats=True)
    assert sum(s["launches"] for s in stats) == 1
    for p, z in zip(probs, zs):
        t, d = p["terms"], p["dets"]
        args = (14, t.flip, t.phase, t.cf, d.idx, d.cf)
        want = (oracle_lib.trott(*args, 1, 0.1) if kind == "trott" else
                oracle_lib.qdrift(*args, 1, 16, 0.05, p["seed"]))
        assert np.array_equal(z, want)


@pytest.mark.parametrize("count", [32, 74, 75])
def test_fp32_equals_streams(count):
    probs = _problems(count)
    p2.set_precision(p2.PREC_FP32)
    got = p2.batch("trott2", probs)
    p2.set_batch_persistent(False)
    for a, b in zip(got, p2.batch("trott2", probs)):
        assert np.array_equal(a, b)
