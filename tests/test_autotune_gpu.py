"""The autotuner's probes run the pass kernels that its table steers: one
launch and one state round trip a pass, no kept plans (at a width beyond the
graphs'), and as many passes as runs of probe rotations."""

import ctypes as C

import pytest

import phase2_b200 as p2
from phase2_b200 import autotune

pytestmark = pytest.mark.gpu


def test_probes_run_pass_kernels(monkeypatch):
    p2.world_ensure()
    seen = []
    real = autotune._time_passes

    def timed(reg, flip, phase, phi):
        out = real(reg, flip, phase, phi)
        seen.append((reg.stats(), len(flip)))
        return out

    monkeypatch.setattr(autotune, "_time_passes", timed)
    lib = p2.lib()
    saved = {}
    for prec in (0, 1):
        for m in range(6):
            v, s = C.c_int(), C.c_int()
            lib.phase2_tune_get(prec, m, C.byref(v), C.byref(s))
            saved[prec, m] = v.value, s.value
    try:
        autotune.sweep_launch(25, groups=6, reps=1)
    finally:
        for (prec, m), e in saved.items():
            lib.phase2_tune_set(prec, m, *e)
    assert seen
    for st, n in seen:
        assert st["sweeps"] == st["passes"] == st["launches"]
        assert st["graph_replays"] == 0
        assert n % st["passes"] == 0
