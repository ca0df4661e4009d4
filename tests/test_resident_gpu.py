"""Registers whose passes run as sub-passes (held on chip up to 14 qubits, a
tile a block up to 19): the oracle's bits at the widths where the kernel or
the block count changes, every span, long sub-passes, and more plans than
the register keeps."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import Register, workloads

pytestmark = pytest.mark.gpu


def _rots(n, k, seed):
    """Runs of equal strings (long sub-passes), groups and dense strings."""
    rng = np.random.Generator(np.random.PCG64(seed))
    t = workloads.random_terms(n, k, seed=seed)
    t.flip[: k // 2] = t.flip[0]
    t.phase[: k // 4] = t.phase[0]
    t.flip[rng.random(k) < 0.1] = 0
    return t.flip, t.phase, rng.uniform(-4, 4, k)


@pytest.mark.parametrize("n", [3, 4, 8, 11, 12, 13, 14, 15, 17, 19, 20])
def test_bits_and_plans(n, oracle_lib):
    rng = np.random.Generator(np.random.PCG64(n))
    amp = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    amp /= np.linalg.norm(amp)
    sets = [_rots(n, 300 if k == 0 else 30, 100 * n + k) for k in range(11)]
    with Register(n, p2.PREC_FP64) as r:
        r.set_state(amp)
        for k in (0, 0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 0, 3, 3):
            r.paulirot(*sets[k])
            r.synchronize()
            amp = oracle_lib.rotate(amp, n, *sets[k])
        assert np.array_equal(r.get_state(), amp)


@pytest.mark.parametrize("n", [5, 11, 13, 14, 15, 19])
def test_forms_share_a_register(n, oracle_lib):
    """Flushes of the FP32-arithmetic form (pass kernels, replayed from
    graphs) and of the mixed form (on chip) take turns on one register's
    plan slots."""
    flip, phase, phi = _rots(n, 60, n)
    phi = 0.01 * phi
    amp = np.zeros(1 << n, dtype=np.complex128)
    amp[1] = 1.0
    old = p2.get_fp32_form()
    try:
        with Register(n, p2.PREC_FP32) as r:
            r.set_state(amp)
            for k in range(24):
                p2.set_fp32_form(p2.FORM_LIFTED_F32 if k % 4 < 2
                                 else p2.FORM_LIFTED_MIXED)
                m = 60 - k // 2
                r.paulirot(flip[:m], phase[:m], phi[:m])
                r.synchronize()
                amp = oracle_lib.rotate(amp, n, flip[:m], phase[:m], phi[:m])
            assert np.max(np.abs(r.get_state() - amp)) < 1e-5
    finally:
        p2.set_fp32_form(old)


@pytest.mark.parametrize("fusion", [(1, 1), (2, 0), (4, 3)])
@pytest.mark.parametrize("n", [10, 14, 16, 19])
def test_spans(n, fusion, oracle_lib):
    flip, phase, phi = _rots(n, 80, 7 * n)
    amp = np.zeros(1 << n, dtype=np.complex128)
    amp[5] = 1.0
    with Register(n, p2.PREC_FP64) as r:
        r.set_fusion(*fusion)
        r.set_state(amp)
        r.paulirot(flip, phase, phi)
        assert np.array_equal(r.get_state(),
                              oracle_lib.rotate(amp, n, flip, phase, phi))
