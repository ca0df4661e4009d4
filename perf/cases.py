"""Performance cases: the calls a user of this package makes, over the
range of sizes it is used at.

The package evolves a 2^n-amplitude state by Pauli rotations (product
formulas of a chemistry Hamiltonian) and reads overlaps.  Its inputs are
host arrays (terms, determinants, angles) and its outputs are host values,
so the whole call, through the Python entry points, is what counts.  Inputs
are synthetic: Jordan-Wigner-like excitation strings with log-uniform
coefficients (or uniformly random strings), determinants of half filling.

``exact`` evolves the same inputs in complex128 with plain torch, without
this package.
"""

from __future__ import annotations

import itertools
import math

import numpy as np
import torch

import phase2_b200 as p2

FP64, FP32 = "fp64", "fp32"
_PREC = {FP64: p2.PREC_FP64, FP32: p2.PREC_FP32}
_ORDER = {"lex": 0, "given": 1, "flip": 2}
_ELEM = {FP64: 16, FP32: 8}


def listed():
    return [
        # one-shot call on text strings: a small molecule's Hamiltonian,
        # once (a script or a notebook cell); latency of the whole call
        dict(name="run-10q", kind="run", nqb=10, nterms=251, prec=FP64,
             delta=0.1),
        # dense random strings on a small register, a few Trotter steps,
        # final state kept: method development and checks
        dict(name="trott-12q", kind="trott", nqb=12, nterms=200, steps=4,
             prec=FP64, strings="random", ndets=1, delta=0.1, order="lex",
             keep_state=True),
        # many short stochastic samples of a small molecule
        dict(name="qdrift-10q", kind="qdrift", nqb=10, nterms=251,
             samples=64, depth=300, prec=FP64, ndets=1, step_size=0.05),
        # the same in the FP32 state, a larger active space
        dict(name="qdrift-14q-fp32", kind="qdrift", nqb=14, nterms=1000,
             samples=32, depth=1000, prec=FP32, ndets=1, step_size=0.05),
        # a correlated trial state (coefficient matrix): expansion, a few
        # second-order steps, overlap with the whole expansion
        dict(name="coeff-16q", kind="coeff", nqb=16, nterms=500, steps=4,
             prec=FP64, delta=0.05, order="lex"),
        # the register API by hand: upload a state, rotate, norm, inner
        # product with a dense trial, download (17 qubits: an odd width)
        dict(name="register-17q", kind="register", nqb=17, nterms=600,
             prec=FP64, delta=0.05),
        # second-order Trotter at a width that fits the L2 cache
        dict(name="trott2-20q-fp32", kind="trott2", nqb=20, nterms=300,
             steps=10, prec=FP32, strings="jw", ndets=2, delta=0.05,
             order="lex", keep_state=False),
        # independent problems of uneven size in one launch
        dict(name="batch-fp32", kind="batch", lo=14, hi=20, count=10,
             terms_lo=100, terms_hi=1500, steps=4, prec=FP32, delta=0.05),
        # composite integrator: heaviest terms deterministic, rest sampled
        dict(name="cmpsit-24q", kind="cmpsit", nqb=24, nterms=4000,
             length=150, depth=350, steps=2, samples=1, prec=FP64, ndets=4),
        # a long Hamiltonian sorted by flip mask: many rotations per sweep
        dict(name="trott2-26q-flip-fp32", kind="trott2", nqb=26,
             nterms=2000, steps=1, prec=FP32, strings="jw", ndets=16,
             delta=0.05, order="flip", keep_state=False),
        # double precision beyond every cache
        dict(name="qdrift-28q", kind="qdrift", nqb=28, nterms=20000,
             samples=1, depth=512, prec=FP64, ndets=1, step_size=1e-3),
        # the largest register of everyday use: 8 GiB of FP32 amplitudes
        dict(name="qdrift-30q-fp32", kind="qdrift", nqb=30, nterms=20000,
             samples=1, depth=256, prec=FP32, ndets=1, step_size=1e-3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds: widths over the whole range, term
    counts and lengths log-uniform, cut to at most the largest case's work
    (2^38 rotation-amplitudes)."""
    kind = rng.choice(["run", "trott", "trott", "trott2", "trott2", "qdrift",
                       "qdrift", "cmpsit", "coeff", "register", "batch"])
    prec = rng.choice([FP64, FP32])
    budget = 2.0 ** 36
    if kind == "run":
        return dict(kind=kind, nqb=rng.randint(4, 20),
                    nterms=_log_int(rng, 20, 1500), prec=FP64, delta=0.1)
    if kind == "coeff":
        return dict(kind=kind, nqb=2 * rng.randint(5, 10),
                    nterms=_log_int(rng, 50, 800), steps=rng.randint(1, 5),
                    prec=prec, delta=0.05, order="lex")
    if kind == "register":
        return dict(kind=kind, nqb=rng.randint(6, 21),
                    nterms=_log_int(rng, 50, 2000), prec=prec, delta=0.05)
    if kind == "batch":
        lo = rng.randint(8, 16)
        return dict(kind=kind, lo=lo, hi=lo + rng.randint(2, 5),
                    count=rng.randint(3, 12), terms_lo=50,
                    terms_hi=_log_int(rng, 100, 1000),
                    steps=rng.randint(1, 5), prec=prec, delta=0.05)
    nqb = rng.randint(8, 28)
    rots = int(min(40000, max(100, budget / 2.0 ** nqb)))
    if kind in ("trott", "trott2"):
        steps = rng.randint(1, 6)
        nterms = max(20, min(_log_int(rng, 100, 6000), rots // (2 * steps)))
        return dict(kind=kind, nqb=nqb, nterms=nterms, steps=steps, prec=prec,
                    strings=rng.choice(["jw", "jw", "random"]),
                    ndets=rng.choice([1, 1, 2, 16]), delta=0.05,
                    order=rng.choice(["lex", "lex", "flip"]),
                    keep_state=nqb <= 14 and rng.random() < 0.5)
    if kind == "qdrift":
        depth = _log_int(rng, 50, max(60, min(2000, rots)))
        samples = max(1, min(rng.randint(1, 64), rots // depth))
        return dict(kind=kind, nqb=nqb, nterms=_log_int(rng, 200, 20000),
                    samples=samples, depth=depth, prec=prec,
                    ndets=rng.choice([1, 1, 2]),
                    step_size=rng.choice([1e-3, 0.05]))
    steps = rng.randint(1, 3)
    half = max(40, min(1000, rots // (2 * steps)))
    length = rng.randint(10, half // 2)
    return dict(kind="cmpsit", nqb=nqb,
                nterms=length + _log_int(rng, 100, 4000), length=length,
                depth=half - length, steps=steps, samples=1, prec=prec,
                ndets=rng.choice([1, 4]))


# ---- inputs ------------------------------------------------------------


def _chain(lo, hi):
    """Z on every qubit strictly between lo < hi."""
    one = np.uint64(1)
    return ((one << hi) - one) & ~((one << (lo + one)) - one)


def _jw(nqb, nterms, rng):
    """Jordan-Wigner-like strings: 9 in 10 two-body groups (8 strings with
    an even number of Y on p<q<r<s), 1 in 10 one-body pairs (XX, YY on
    p<q), Z chains between; then a tenth of the terms diagonal (Z, ZZ).
    Coefficients +-10^U(-6, 0)."""
    n_z = nterms // 10
    n = nterms - n_z
    sel = max(1, n // 2)
    pos = np.sort(np.argsort(rng.random((sel, nqb)), axis=1)[:, :4],
                  axis=1).astype(np.uint64)
    two = rng.random(sel) >= 0.1
    bit = np.uint64(1) << pos
    xy8 = np.array([v for v in itertools.product((0, 1), repeat=4)
                    if sum(v) % 2 == 0], dtype=np.uint64)
    f2 = bit.sum(axis=1, dtype=np.uint64)
    z2 = _chain(pos[:, 0], pos[:, 1]) | _chain(pos[:, 2], pos[:, 3])
    f1 = bit[:, 0] | bit[:, 1]
    z1 = _chain(pos[:, 0], pos[:, 1])
    flip, phase = [], []
    for k in range(sel):
        if two[k]:
            flip.append(np.full(8, f2[k]))
            phase.append(z2[k] | (xy8 * bit[k]).sum(axis=1, dtype=np.uint64))
        else:
            flip.append(np.full(2, f1[k]))
            phase.append(z1[k] | np.array([0, f1[k]], dtype=np.uint64))
    flip = np.concatenate(flip)[:n]
    phase = np.concatenate(phase)[:n]
    a = rng.integers(0, nqb, size=n_z).astype(np.uint64)
    b = rng.integers(0, nqb, size=n_z).astype(np.uint64)
    zz = (np.uint64(1) << a) | (np.uint64(1) << b)
    flip = np.concatenate([flip, np.zeros(n_z, dtype=np.uint64)])
    phase = np.concatenate([phase, zz])
    m = len(flip)
    cf = 10.0 ** rng.uniform(-6.0, 0.0, size=m)
    cf *= np.where(rng.random(m) < 0.5, -1.0, 1.0)
    return flip, phase, cf


def _random(nqb, nterms, rng):
    """Every qubit's operator uniform over I, X, Y, Z."""
    ops = rng.integers(0, 4, size=(nterms, nqb))
    bit = np.uint64(1) << np.arange(nqb, dtype=np.uint64)
    flip = ((ops == 1) | (ops == 2)).astype(np.uint64) @ bit
    phase = (ops >= 2).astype(np.uint64) @ bit
    return flip, phase, rng.standard_normal(nterms) / math.sqrt(nterms)


def _dets(nqb, ndets, rng):
    """ndets distinct determinants of weight nqb // 2, normalised."""
    ndets = min(ndets, math.comb(nqb, nqb // 2))
    seen = {}
    while len(seen) < ndets:
        occ = rng.permutation(nqb)[:nqb // 2]
        seen[int(sum(1 << int(q) for q in occ))] = None
    cf = rng.standard_normal(ndets) + 1j * rng.standard_normal(ndets)
    cf /= np.linalg.norm(cf)
    if ndets == 1:
        cf = np.ones(1, dtype=np.complex128)
    return np.array(list(seen), dtype=np.uint64), cf


def _text(flip, phase, nqb):
    out = []
    for f, z in zip(flip.tolist(), phase.tolist()):
        s = []
        for q in range(nqb):
            op = (f >> q & 1) | (z >> q & 1) << 1
            if op:
                s.append("IXZY"[op] + str(q))
        out.append(" ".join(s))
    return out


def _batch_sizes(case):
    """(qubits, terms, steps) of every instance: widths, term counts and
    step counts spread over their ranges, out of step with one another."""
    out = []
    n = case["count"]
    for k in range(n):
        nqb = case["lo"] + 7 * k % (case["hi"] - case["lo"] + 1)
        at = (3 * k % n) / max(1, n - 1)
        nt = case["terms_lo"] * (case["terms_hi"] / case["terms_lo"]) ** at
        out.append((nqb, int(round(nt)), 1 + 5 * k % case["steps"]))
    return out


def _inputs(case, seed):
    """Every input of a case, as plain numpy arrays."""
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    kind = case["kind"]
    if kind == "batch":
        return dict(problems=[
            dict(nqb=nqb, terms=_jw(nqb, nt, rng), dets=_dets(nqb, 1, rng),
                 steps=steps, delta=case["delta"])
            for nqb, nt, steps in _batch_sizes(case)])
    nqb = case["nqb"]
    make = _random if case.get("strings") == "random" else _jw
    d = dict(terms=make(nqb, case["nterms"], rng))
    if kind == "run":
        d["psi"] = "".join(rng.permutation(
            ["1"] * (nqb // 2) + ["0"] * (nqb - nqb // 2)).tolist())
    elif kind == "coeff":
        m, k = nqb // 2, max(1, nqb // 4)
        q, _ = np.linalg.qr(rng.standard_normal((m, m)))
        d["orb"] = np.ascontiguousarray(q[:, :k])
    elif kind == "register":
        for key in ("psi", "trial"):
            v = rng.standard_normal(1 << nqb) + 1j * rng.standard_normal(
                1 << nqb)
            d[key] = v / np.linalg.norm(v)
    else:
        d["dets"] = _dets(nqb, case["ndets"], rng)
    if kind in ("qdrift", "cmpsit"):
        d["seed"] = int(rng.integers(1, 1 << 62))
    if kind == "cmpsit":
        lam = float(np.sort(np.abs(d["terms"][2]))[::-1]
                    [case["length"]:].sum())
        d["angle_rand"] = 0.05 * lam / case["depth"]
    return d


def prepare(case, seed):
    """The Hamiltonian, trial state and (register case) the register that a
    program holds before the call."""
    p2.world_ensure()
    s = dict(case=dict(case), **_inputs(case, seed))
    kind = case["kind"]
    if kind == "run":
        s["text"] = _text(s["terms"][0], s["terms"][1], case["nqb"])
        s["coeffs"] = s["terms"][2].tolist()
    elif kind == "batch":
        s["problems"] = [dict(p, terms=p2.Terms(*p["terms"]),
                              dets=p2.Dets(*p["dets"]))
                         for p in s["problems"]]
    else:
        if kind == "coeff":
            n = case["nqb"] // 2
            k = s["orb"].shape[1]
            s["trial"] = p2.CoeffMatrix(n, k, k, [s["orb"]])
        elif kind == "register":
            s["phi"] = case["delta"] * s["terms"][2]
            s["reg"] = p2.Register(case["nqb"], _PREC[case["prec"]])
        else:
            s["trial"] = p2.Dets(*s["dets"])
        s["ham"] = p2.Terms(*s["terms"])
    return s


def run(state):
    c = state["case"]
    kind = c["kind"]
    p2.set_precision(_PREC[c["prec"]])
    if kind == "run":
        return np.array(p2.run(state["text"], state["coeffs"], c["delta"],
                               state["psi"]))
    if kind == "register":
        reg, t = state["reg"], state["ham"]
        reg.set_state(state["psi"])
        reg.paulirot(t.flip, t.phase, state["phi"])
        norm = reg.norm2()
        z = reg.inner_dense(state["trial"])
        return norm, np.array(z), reg.get_state()
    p2.set_term_order(_ORDER[c.get("order", "lex")])
    if kind == "batch":
        return p2.batch("trott", state["problems"])
    if kind == "coeff":
        return p2.trott2(c["nqb"], state["ham"], state["trial"], c["steps"],
                         c["delta"])
    if kind == "qdrift":
        return p2.qdrift(c["nqb"], state["ham"], state["trial"],
                         c["samples"], c["depth"], c["step_size"],
                         state["seed"])
    if kind == "cmpsit":
        return p2.cmpsit(c["nqb"], state["ham"], state["trial"],
                         c["samples"], c["steps"], c["length"], c["depth"],
                         0.05, state["angle_rand"], state["seed"])
    step = p2.trott if kind == "trott" else p2.trott2
    if c["keep_state"]:
        vals, stats = step(c["nqb"], state["ham"], state["trial"],
                           c["steps"], c["delta"], with_stats=True,
                           with_state=True)
        return vals, stats["state"]
    return step(c["nqb"], state["ham"], state["trial"], c["steps"],
                c["delta"])


# ---- work --------------------------------------------------------------


def _rotations(case):
    """(rotations, outputs) of one pass of a case other than a batch."""
    kind = case["kind"]
    if kind in ("run", "register"):
        return case["nterms"], 1
    if kind in ("trott", "trott2", "coeff"):
        per = case["nterms"] * (1 if kind == "trott" else 2)
        return per * case["steps"], case["steps"]
    if kind == "qdrift":
        return case["samples"] * case["depth"], case["samples"]
    return (case["samples"] * 2 * case["steps"] *
            (case["length"] + case["depth"]), case["samples"])


def work(case):
    """A rotation is 6 operations an amplitude (two complex scalings by real
    numbers and their sum); every output needs the state read and written
    at least once (a step or sample depends on all of it), and every term
    is read once."""
    if case["kind"] == "batch":
        sizes = _batch_sizes(case)
        return {"bytes": sum(2.0 ** (n + 1) * _ELEM[case["prec"]] * s +
                             24 * t for n, t, s in sizes),
                "flops": sum(6 * 2.0 ** n * t * s for n, t, s in sizes)}
    rots, outs = _rotations(case)
    amps = 2.0 ** case["nqb"]
    more = 0.0
    if case["kind"] == "register":
        # state and trial in, state out, at 16 bytes
        more = 48 * amps
    elif case.get("keep_state"):
        more = 16 * amps
    return {"bytes": 2 * amps * _ELEM[case["prec"]] * outs +
            24 * case["nterms"] + more,
            "flops": 6 * amps * rots}


# ---- 64-bit values -----------------------------------------------------


class _State:
    """2^n complex128 amplitudes as a 2-D array (high bits, low bits), on
    the GPU where there is one."""

    def __init__(self, nqb):
        self.lo = nqb // 2
        self.hi = nqb - self.lo
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.ih = torch.arange(1 << self.hi, device=self.dev)
        self.il = torch.arange(1 << self.lo, device=self.dev)
        self.a = torch.zeros((1 << self.hi, 1 << self.lo),
                             dtype=torch.complex128, device=self.dev)

    def _split(self, m):
        return int(m) >> self.lo, int(m) & ((1 << self.lo) - 1)

    @staticmethod
    def _sign(idx, mask):
        v = idx & mask
        for s in (32, 16, 8, 4, 2, 1):
            v = v ^ (v >> s)
        return 1.0 - 2.0 * (v & 1).to(torch.float64)

    def set(self, idx, z):
        self.a.zero_()
        for i, v in zip(idx, z):
            h, q = self._split(i)
            self.a[h, q] = complex(v)

    def rotate(self, flip, phase, phi):
        """a_g <- cos(phi) a_g + i sin(phi) conj(z_g) a_(g ^ flip), z_g =
        i^(|flip & phase| + 2 |g & phase|)."""
        fh, fl = self._split(flip)
        zh, zl = self._split(phase)
        k = bin(int(flip) & int(phase)).count("1") & 3
        coef = 1j * math.sin(phi) * (1, -1j, -1, 1j)[k]
        sh = self._sign(self.ih, zh)[:, None]
        sl = (self._sign(self.il, zl) * coef)[None, :]
        p = self.a
        if fh:
            p = p.index_select(0, self.ih ^ fh)
        if fl:
            p = p.index_select(1, self.il ^ fl)
        p = p.mul(sh) if p is self.a else p.mul_(sh)
        self.a.mul_(math.cos(phi)).add_(p.mul_(sl))

    def dot(self, idx, z):
        tot = 0j
        for i, v in zip(idx, z):
            h, q = self._split(i)
            tot += complex(self.a[h, q].item()) * complex(v).conjugate()
        return tot

    def flat(self):
        return self.a.reshape(-1).cpu().numpy().copy()


def _lex(flip, phase):
    """Order by the Pauli operators (I < X < Y < Z) from the top qubit."""
    def key(k):
        f, z = int(flip[k]), int(phase[k])
        return tuple((0, 1, 3, 2)[(f >> q & 1) | (z >> q & 1) << 1]
                     for q in range(63, -1, -1))
    return sorted(range(len(flip)), key=key)


def _ordered(terms, order):
    flip, phase, cf = terms
    if order == "lex":
        o = _lex(flip, phase)
    elif order == "flip":
        o = np.lexsort((phase, flip))
    else:
        return terms
    return flip[o], phase[o], cf[o]


class _Xoshiro:
    """xoshiro256** seeded by splitmix64, 128 outputs skipped; uniforms are
    the top 53 bits."""
    M = (1 << 64) - 1

    def __init__(self, seed):
        x, s = seed, []
        for _ in range(4):
            x = (x + 0x9e3779b97f4a7c15) & self.M
            z = x
            z = ((z ^ (z >> 30)) * 0xbf58476d1ce4e5b9) & self.M
            z = ((z ^ (z >> 27)) * 0x94d049bb133111eb) & self.M
            s.append(z ^ (z >> 31))
        self.s = s
        for _ in range(128):
            self.next()

    def _rol(self, v, k):
        return ((v << k) | (v >> (64 - k))) & self.M

    def next(self):
        s = self.s
        out = (self._rol((s[1] * 5) & self.M, 7) * 9) & self.M
        t = (s[1] << 17) & self.M
        s[2] ^= s[0]
        s[3] ^= s[1]
        s[1] ^= s[2]
        s[0] ^= s[3]
        s[2] ^= t
        s[3] = self._rol(s[3], 45)
        return out

    def draws(self, n):
        return np.array([(self.next() >> 11) * 2.0 ** -53
                         for _ in range(n)])


def _cdf(cf):
    w = np.abs(cf)
    return np.cumsum(w / np.cumsum(w)[-1])


def _pick(rng, y, n):
    k = np.searchsorted(y, rng.draws(n), side="right")
    return np.minimum(k, len(y) - 1)


def _sign(cf):
    return np.where(np.abs(cf) < np.finfo(np.float64).eps, 0.0, np.sign(cf))


def _trott(st, terms, steps, delta, order2, measure):
    flip, phase, cf = terms
    out = []
    seq = list(range(len(cf)))
    half = delta / 2 if order2 else delta
    seq = seq + seq[::-1] if order2 else seq
    for _ in range(steps):
        for k in seq:
            st.rotate(flip[k], phase[k], half * cf[k])
        out.append(measure())
    return np.array(out)


def exact(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    if kind == "batch":
        if sum(2.0 ** p["nqb"] * len(p["terms"][2]) * p["steps"]
               for p in d["problems"]) > 2.0 ** 35:
            return None
        out = []
        for p in d["problems"]:
            st = _State(p["nqb"])
            st.set(*p["dets"])
            out.append(_trott(st, _ordered(p["terms"], "lex"), p["steps"],
                              p["delta"], False,
                              lambda: st.dot(*p["dets"])))
        return out
    rots, _ = _rotations(case)
    # about 10 s: launches of small states, memory traffic of large ones
    if rots > 60000 or 2.0 ** case["nqb"] * rots > 2.0 ** 38.1:
        return None
    nqb, st = case["nqb"], _State(case["nqb"])
    flip, phase, cf = d["terms"]
    if kind == "run":
        b = sum(1 << k for k, ch in enumerate(d["psi"]) if ch == "1")
        st.set([b], [1.0])
        for k in range(len(cf)):
            st.rotate(flip[k], phase[k], case["delta"] * cf[k])
        return np.array(st.dot([b], [1.0]))
    if kind == "register":
        st.a.copy_(torch.from_numpy(d["psi"]).reshape(st.a.shape))
        for k in range(len(cf)):
            st.rotate(flip[k], phase[k], case["delta"] * cf[k])
        v = st.flat()
        return (float(np.vdot(v, v).real), np.array(np.vdot(d["trial"], v)), v)
    if kind == "coeff":
        m, k = nqb // 2, d["orb"].shape[1]
        subs = list(itertools.combinations(range(m), k))
        det = np.linalg.det(d["orb"][np.array(subs)])
        occ = np.array([sum(1 << q for q in s) for s in subs])
        full = np.zeros(1 << nqb, dtype=np.complex128)
        amp = det[:, None] * det[None, :]
        amp[np.abs(amp) < 1e-12] = 0.0
        full[occ[:, None] | (occ[None, :] << m)] = amp
        trial = torch.from_numpy(full).reshape(st.a.shape).to(st.dev)
        st.a.copy_(trial)
        return _trott(st, _ordered(d["terms"], "lex"), case["steps"],
                      case["delta"], True,
                      lambda: complex((trial.conj() * st.a).sum().item()))
    idx, z = d["dets"]
    if kind in ("trott", "trott2"):
        st.set(idx, z)
        vals = _trott(st, _ordered(d["terms"], case["order"]), case["steps"],
                      case["delta"], kind == "trott2",
                      lambda: st.dot(idx, z))
        return (vals, st.flat()) if case["keep_state"] else vals
    rng = _Xoshiro(d["seed"])
    out = []
    if kind == "qdrift":
        y, omega = _cdf(cf), math.asin(case["step_size"])
        sg = _sign(cf)
        for _ in range(case["samples"]):
            st.set(idx, z)
            for k in _pick(rng, y, case["depth"]):
                st.rotate(flip[k], phase[k], omega * sg[k])
            out.append(st.dot(idx, z))
        return np.array(out)
    o = np.argsort(-np.abs(cf), kind="stable")
    head, rest = o[:case["length"]], o[case["length"]:]
    hf, hz, hc = _ordered((flip[head], phase[head], cf[head]), "lex")
    y, sg = _cdf(cf[rest]), _sign(cf[rest])
    for _ in range(case["samples"]):
        st.set(idx, z)
        for half in range(2 * case["steps"]):
            k = _pick(rng, y, case["depth"])
            f = np.concatenate([hf, flip[rest][k]])
            p = np.concatenate([hz, phase[rest][k]])
            a = np.concatenate([0.5 * (hc * 0.05),
                                0.5 * (sg[k] * d["angle_rand"])])
            seq = range(len(a)) if half % 2 == 0 else range(len(a) - 1, -1,
                                                            -1)
            for j in seq:
                st.rotate(f[j], p[j], a[j])
        out.append(st.dot(idx, z))
    return np.array(out)
