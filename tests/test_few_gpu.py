"""Amplitude writes and reads passed with a launch: both sides of the limit,
repeated indices (the later write holds), reads before and after a change,
and in either precision."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import Register

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [p2.PREC_FP64, p2.PREC_FP32])
@pytest.mark.parametrize("n", [6, 12, 18])
@pytest.mark.parametrize("k", [1, 31, 32, 33, 64])
def test_writes_and_reads(k, n, prec):
    rng = np.random.Generator(np.random.PCG64(k * n))
    idx = rng.integers(0, 1 << n, k, dtype=np.uint64)
    idx[-1] = idx[0]
    z = (rng.standard_normal(k) + 1j * rng.standard_normal(k)).astype(
        np.complex64).astype(np.complex128)
    want = np.zeros(1 << n, dtype=np.complex128)
    for i, v in zip(idx, z):
        want[i] = v
    with Register(n, prec) as r:
        r.setamps(idx, z)
        for m in (1, k, k):
            assert np.array_equal(r.getamps(idx[:m]), want[idx[:m]])
        r.zero()
        assert not np.any(r.getamps(idx))
        r.setamps(idx[:1], z[:1])
        want[:] = 0
        want[idx[0]] = z[0]
        assert np.array_equal(r.getamps(idx), want[idx])
        assert np.array_equal(r.get_state(), want)
        assert abs(r.norm2() - abs(z[0]) ** 2) < 1e-12
