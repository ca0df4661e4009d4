"""Reads of registers that keep a host copy: a zeroed register and a narrow
one's second read start no further copy, and every read is the state's."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import Register

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _world():
    p2.world_ensure()


@pytest.mark.parametrize("prec", [p2.PREC_FP64, p2.PREC_FP32])
@pytest.mark.parametrize("n", [1, 9, 10, 12, 13, 16])
def test_copies_and_values(n, prec):
    rng = np.random.Generator(np.random.PCG64(n))
    amp = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    amp = amp.astype(np.complex64).astype(np.complex128)
    last = (1 << n) - 1

    def copies(r):
        st = r.stats()
        return st["launches"], st["d2h_bytes"]

    with Register(n, prec) as r:
        r.set_state(amp)
        assert r.getamps([last])[0] == amp[last]
        first = copies(r)
        assert np.array_equal(r.getamps([0, last]), amp[[0, last]])
        if n < 10:
            assert copies(r) == first
        second = copies(r)
        assert np.array_equal(r.get_state(), amp)
        assert r.getamps([last])[0] == amp[last]
        assert copies(r) == second
        r.zero()
        before = copies(r)
        assert not r.getamps([0, last]).any()
        assert not r.get_state().any()
        assert not r.getamps(np.zeros(50, dtype=np.uint64)).any()
        assert copies(r) == before
        r.setamps([last], [2.0])
        assert r.getamps([last])[0] == 2.0
        r.set_state(amp)
        assert np.array_equal(r.get_state(), amp)
