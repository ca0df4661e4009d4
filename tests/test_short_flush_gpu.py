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
