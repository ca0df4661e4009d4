"""Registers that take over a destroyed register's stream and buffers start
as new ones: zero state, no counters, no timing, no plans; from several
threads at once too."""

import threading

import numpy as np
import pytest

import phase2_b200 as p2
from phase2_b200 import Register, workloads

pytestmark = pytest.mark.gpu


def _use(n, prec, oracle_lib, out, k):
    t = workloads.random_terms(n, 40, seed=n)
    phi = np.linspace(-1, 1, 40)
    amp = np.zeros(1 << n, dtype=np.complex128)
    amp[3] = 1.0
    want = oracle_lib.rotate(amp, n, t.flip, t.phase, phi)
    ok = True
    for rep in range(4):
        with Register(n, prec) as r:
            st = r.stats()
            ok = ok and not any(st.values())
            ok = ok and not np.any(r.get_state())
            r.setamps([3], [1.0])
            if rep == 1:
                r.set_timing(True)
            r.paulirot(t.flip, t.phase, phi)
            got = r.get_state()
            tol = 0 if prec == p2.PREC_FP64 else 1e-5
            ok = ok and np.max(np.abs(got - want)) <= tol
            if rep != 1:
                ok = ok and r.stats()["pass_ms"] == 0
    out[k] = ok


def test_reused_shells(oracle_lib):
    sizes = [(4, 0), (11, 0), (13, 1), (17, 0), (17, 1), (18, 1)]
    out = [False] * len(sizes)
    for k, (n, prec) in enumerate(sizes):
        _use(n, prec, oracle_lib, out, k)
    assert all(out), out
    out = [False] * len(sizes)
    th = [threading.Thread(target=_use, args=(n, prec, oracle_lib, out, k))
          for k, (n, prec) in enumerate(sizes)]
    for x in th:
        x.start()
    for x in th:
        x.join()
    assert all(out), out
