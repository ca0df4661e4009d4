"""Sign variants of the FP64-arithmetic shears (pass kernels, 20 qubits up):
the bits of the sub-passes that run a 19-qubit register, whose kernel takes
every sign at run time, on the same state below a zero upper half."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import Register

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("span", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("low", [0, 7])
def test_bits(span, low):
    n = 19
    rng = np.random.Generator(np.random.PCG64(10 * span + low))
    # masks whose span stays one pass, its pivots from bit `low` up
    rows = rng.integers(1, 1 << (n - low), size=span).astype(np.uint64)
    rows <<= np.uint64(low)
    pick = rng.integers(0, 2, size=(200, span)).astype(bool)
    flip = np.array([np.bitwise_xor.reduce(rows[p]) if p.any() else 0
                     for p in pick], dtype=np.uint64)
    phase = rng.integers(0, 1 << n, size=200).astype(np.uint64)
    phi = rng.uniform(-4, 4, 200)
    amp = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    amp = (amp / np.linalg.norm(amp)).astype(np.complex64)
    with Register(n, p2.PREC_FP32) as a, Register(n + 1, p2.PREC_FP32) as b:
        a.set_state(amp.astype(np.complex128))
        b.set_state(np.concatenate([amp, 0 * amp]).astype(np.complex128))
        for r in (a, b):
            r.paulirot(flip, phase, phi)
            r.synchronize()
        got = b.get_state()
        assert np.array_equal(got[: 1 << n], a.get_state())
        assert not got[1 << n:].any()
