"""Tile runs well beyond a wave of tiles (24 qubits): the bits of one
rotation a pass."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import Register, workloads

pytestmark = pytest.mark.gpu


def test_bits():
    p2.world_ensure()
    n = 24
    t = workloads.random_terms(n, 24, seed=n)
    phi = np.linspace(-2, 2, 24)
    rng = np.random.Generator(np.random.PCG64(6))
    amp = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    out = []
    for fusion in ((1, 1), (5, 0)):
        with Register(n, p2.PREC_FP64) as r:
            r.set_fusion(*fusion)
            r.set_state(amp)
            r.paulirot(t.flip, t.phase, phi)
            out.append((r.get_state(), r.stats()))
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1]["sweeps"] == 24
    assert out[1][1]["sweeps"] < out[1][1]["passes"]
