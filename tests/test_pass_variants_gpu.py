"""The launch variants of the pass kernels, at a width and a rotation limit
that no other kernel takes: FP64 the oracle's bits, FP32 with FP64 arithmetic
the same bits for every variant."""

import ctypes as C

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import Register, workloads

pytestmark = pytest.mark.gpu

N = 21


@pytest.fixture
def table():
    p2.world_ensure()
    lib = p2.lib()
    saved = []
    for prec in (0, 1):
        for m in range(6):
            v, s = C.c_int(), C.c_int()
            assert lib.phase2_tune_get(prec, m, C.byref(v), C.byref(s)) == 0
            saved.append((prec, m, v.value, s.value))
    form = p2.get_fp32_form()

    def choose(prec, variant, per_sm):
        for m in range(6):
            assert lib.phase2_tune_set(prec, m, variant, per_sm) == 0
    yield choose
    for e in saved:
        lib.phase2_tune_set(*e)
    p2.set_fp32_form(form)


def _rotations(low, count, seed):
    """Masks from bit `low` up, a fifth of them diagonal."""
    t = workloads.random_terms(N, count, seed=seed)
    t.flip[::5] = 0
    flip = t.flip >> np.uint64(low) << np.uint64(low)
    return flip, t.phase, np.linspace(-3, 3, count)


def _state(seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    a = rng.standard_normal(1 << N) + 1j * rng.standard_normal(1 << N)
    a = (a / np.linalg.norm(a)).astype(np.complex64)
    return a.astype(np.complex128)


def _run(prec, span, amp, ops):
    with Register(N, prec) as r:
        r.set_fusion(span, 40)
        r.set_state(amp)
        r.paulirot(*ops)
        got, st = r.get_state(), r.stats()
    # one launch and one state round trip a pass: the pass kernels
    assert st["launches"] == st["passes"] == st["sweeps"] > 0
    assert st["graph_replays"] == 0
    return got


def test_fp64_variants(table, oracle_lib):
    amp, ops = _state(1), _rotations(0, 24, 2)
    want = oracle_lib.rotate(amp, N, *ops)
    for variant, per_sm in ((0, 0), (1, 0), (0, 4), (1, 2)):
        table(p2.PREC_FP64, variant, per_sm)
        for span in (1, 2, 3, 4, 5):
            assert np.array_equal(_run(p2.PREC_FP64, span, amp, ops), want), (
                variant, per_sm, span)


@pytest.mark.parametrize("form", [p2.FORM_LIFTED, p2.FORM_LIFTED_MIXED])
@pytest.mark.parametrize("low", [0, 5])
def test_fp32_variants(table, low, form, oracle_lib):
    """Masks from bit 5 up are what the staged variants take (spans 3 to 5);
    with lower ones they leave the pass to the direct kernel."""
    p2.set_fp32_form(form)
    amp, ops = _state(3 + low), _rotations(low, 24, 4 + low)
    exact = oracle_lib.rotate(amp, N, *ops)
    for span in (2, 3, 4, 5):
        table(p2.PREC_FP32, 0, 0)
        want = _run(p2.PREC_FP32, span, amp, ops)
        assert np.max(np.abs(want - exact)) < 1e-5
        for variant, per_sm in ((1, 0), (2, 0), (3, 0), (1, 2), (2, 1)):
            table(p2.PREC_FP32, variant, per_sm)
            assert np.array_equal(_run(p2.PREC_FP32, span, amp, ops), want), (
                variant, per_sm, span)
