"""FP64 tile runs: the bits of one rotation a pass, at the narrowest width
and beyond one wave of tiles, for draws, dense strings and diagonal ones;
repeated plans; and the planned passes where those are asked for or long."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import Register, workloads

pytestmark = pytest.mark.gpu


def _strings(n, kind):
    rng = np.random.Generator(np.random.PCG64(n))
    if kind == "draws":
        t = workloads.jw_terms(n, 400, seed=n)
        o = rng.permutation(400)[:90]
        return t.flip[o], t.phase[o]
    t = workloads.random_terms(n, 60, seed=n)
    if kind == "diagonal":
        t.flip[::2] = 0
    if kind == "runs":
        t.flip[1::2] = t.flip[::2]
        f = np.concatenate([t.flip, np.full(140, t.flip[0])])
        z = np.concatenate([t.phase, rng.integers(0, 1 << n, 140,
                                                  dtype=np.uint64)])
        return f, z
    return t.flip, t.phase


@pytest.mark.parametrize("kind", ["draws", "dense", "diagonal", "runs"])
@pytest.mark.parametrize("n", [20, 22])
def test_bits(n, kind):
    flip, phase = _strings(n, kind)
    phi = np.linspace(-2, 2, len(flip))
    rng = np.random.Generator(np.random.PCG64(5))
    amp = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    out = []
    for fusion in ((1, 1), (5, 0)):
        with Register(n, p2.PREC_FP64) as r:
            r.set_fusion(*fusion)
            r.set_state(amp)
            for _ in range(2):
                r.paulirot(flip, phase, phi)
                r.synchronize()
            out.append((r.get_state(), r.stats()))
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1]["sweeps"] == 2 * len(flip)
    st = out[1][1]
    if st["rotations"] <= 10 * st["passes"]:
        assert st["sweeps"] < st["passes"]
    else:  # bound by arithmetic: the planned passes
        assert st["sweeps"] == st["passes"]
    assert out[1][1]["graph_replays"] >= 1
