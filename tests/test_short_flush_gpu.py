"""Flushes of a few rotations: the kernels they are sent to (a plan kept on
the device counts its replays) and their bits, against one rotation a pass."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import Register

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _world():
    p2.world_ensure()


def _flush(n, count, one_mask, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    flip = rng.integers(1, 1 << n, count).astype(np.uint64)
    if one_mask:
        flip[:] = flip[0]
        flip[1::3] = 0
    return (flip, rng.integers(0, 1 << n, count).astype(np.uint64),
            rng.uniform(-3, 3, count))


def _run(n, prec, fusion, ops):
    rng = np.random.Generator(np.random.PCG64(n))
    amp = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    with Register(n, prec) as r:
        r.set_fusion(*fusion)
        r.set_state(amp / np.linalg.norm(amp))
        for op in ops:
            r.paulirot(*op)
            r.synchronize()
        return r.get_state(), r.stats()


# flush, runs it again is given, replays of a kept plan
@pytest.mark.parametrize("count,one_mask,replays", [
    (1, False, 1), (4, True, 1), (6, True, 1),  # one mask: tiles
    (2, False, 0), (5, False, 0), (7, True, 0),  # a pass
    (10, False, 1), (15, False, 1)])  # a graph; tiles
@pytest.mark.parametrize("n", [21, 22])
def test_wide_exact(n, count, one_mask, replays):
    a = _flush(n, count, one_mask, 3 * count)
    got, st = _run(n, p2.PREC_FP64, (5, 0), [a, a])
    want, _ = _run(n, p2.PREC_FP64, (1, 1), [a, a])
    assert np.array_equal(got, want)
    assert st["graph_replays"] == replays


@pytest.mark.parametrize("count", [1, 5, 8])
@pytest.mark.parametrize("n", [3, 5, 10, 11, 13, 14, 15, 19, 20])
def test_narrow(n, count):
    a = _flush(n, count, True, count)
    b = _flush(n, count, True, count + 100)
    # two flushes in turn: pass kernels; the same again: its plan is kept
    turns = [a, b, a, b]
    got, st = _run(n, p2.PREC_FP64, (5, 0), turns)
    assert st["graph_replays"] == 0
    assert np.array_equal(got, _run(n, p2.PREC_FP64, (1, 1), turns)[0])
    again = [a, a, a, b, a]
    got, st = _run(n, p2.PREC_FP64, (5, 0), again)
    assert st["graph_replays"] == 1
    assert np.array_equal(got, _run(n, p2.PREC_FP64, (1, 1), again)[0])


@pytest.mark.parametrize("count", [1, 5, 8, 10])
@pytest.mark.parametrize("n", [5, 11, 14, 17])
def test_fp32_routes_agree(n, count):
    """The second of two equal flushes runs as sub-passes: the bits of the
    pass kernels, which run it on another register."""
    a = _flush(n, count, count < 10, 7 * count)
    first = _run(n, p2.PREC_FP32, (5, 0), [a])[0]
    got = _run(n, p2.PREC_FP32, (5, 0), [a, a])[0]
    with Register(n, p2.PREC_FP32) as r:
        r.set_state(first)
        r.paulirot(*a)
        assert np.array_equal(r.get_state(), got)
