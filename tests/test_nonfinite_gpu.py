"""Infinities and NaN in a register reach the amplitudes that the rotations
connect them with and no others, which keep their bits: the sign steps of the
FP32 kernels multiply coefficients by +-1, never amplitudes."""

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import Register

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _world():
    p2.world_ensure()
    form = p2.get_fp32_form()
    yield
    p2.set_fp32_form(form)


@pytest.mark.parametrize("count", [6, 30])
@pytest.mark.parametrize("n,prec,form", [
    (12, p2.PREC_FP64, 0), (16, p2.PREC_FP64, 0), (20, p2.PREC_FP64, 0),
    (12, p2.PREC_FP32, p2.FORM_LIFTED), (16, p2.PREC_FP32, p2.FORM_LIFTED),
    (20, p2.PREC_FP32, p2.FORM_LIFTED),
    (12, p2.PREC_FP32, p2.FORM_LIFTED_F32),
    (20, p2.PREC_FP32, p2.FORM_LIFTED_F32),
    (24, p2.PREC_FP32, p2.FORM_LIFTED_MIXED)])
def test_stays_in_its_orbit(n, prec, form, count):
    rng = np.random.Generator(np.random.PCG64(n + count))
    rows = rng.integers(1, 1 << n, 7).astype(np.uint64)
    pick = rng.integers(0, 2, (count, 7)).astype(bool)
    flip = np.array([np.bitwise_xor.reduce(rows[p]) if p.any() else 0
                     for p in pick], dtype=np.uint64)
    phase = rng.integers(0, 1 << n, count).astype(np.uint64)
    phi = rng.uniform(0.1, 1.4, count)
    amp = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    amp = (amp / np.linalg.norm(amp)).astype(np.complex64).astype(complex)
    bad = amp.copy()
    at = rng.integers(0, 1 << n, 2).astype(np.uint64)
    bad[at[0]] = complex(np.inf, 0.0)
    bad[at[1]] = complex(0.0, np.nan)
    if prec == p2.PREC_FP32:
        p2.set_fp32_form(form)
    out = []
    for a in (amp, bad):
        with Register(n, prec) as r:
            r.set_state(a)
            for _ in range(2):
                r.paulirot(flip, phase, phi)
                r.synchronize()
            out.append(r.get_state())
    # the orbit: XORs of the masks
    span = np.zeros(1, dtype=np.uint64)
    for row in rows:
        span = np.unique(np.concatenate([span, span ^ row]))
    reach = np.zeros(1 << n, dtype=bool)
    for a in at:
        reach[span ^ a] = True
    assert np.isfinite(out[0]).all()
    assert not np.isfinite(out[1][at]).any()
    assert np.array_equal(out[0][~reach], out[1][~reach])
