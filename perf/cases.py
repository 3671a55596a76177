"""Measured cases of the propagation engine: what a user has it do, through its
public entry points, from a 4-qubit call to a 99-million-term one.

A case is a dict of plain values; `prepare` makes its inputs from a seed,
`run` makes one pass, `exact` gives what the pass returns from a plain numpy
restatement in 64 bits.  Circuits are the ones of propaq_b200.workloads, with
angles drawn per seed around the stated ones.

Left out of the outputs: PropagationResult.sparse_key_bytes, the device bytes
the engine holds at that moment, which depend on what it ran before.
"""

from __future__ import annotations

import math

import numpy as np

import propaq_b200 as pq
from propaq_b200 import _native, workloads
from propaq_b200.adjoint import ParametrizedExpectation
from propaq_b200.circuits import PauliCircuit, PauliRotation
from propaq_b200.datatypes import PauliString, PauliTermSum
from propaq_b200.propagators import expectation_values, heisenberg_gates, state_words


def listed():
    return [
        # The smallest call: the 4-qubit, 40-rotation noisy circuit of the
        # plugin notebooks; launches, copies and host work are all of it.
        {"name": "register_4q", "kind": "register", "n": 4, "gates": 40, "max_weight": 3, "min_coeff": 1e-4,
         "damping": 0.01},
        # A 20-qubit Trotterised chain, generic angles, no noise (1-word keys,
        # up to 31k terms): the everyday simulation.
        {"name": "tfim_20q", "kind": "tfim", "n": 20, "steps": 10, "max_weight": 8, "min_coeff": 1e-4},
        # The noisy kicked-Ising benchmark on 100 qubits (4-word keys).
        {"name": "kicked_10x10", "kind": "kicked", "rows": 10, "cols": 10, "steps": 20, "theta": 0.6, "p": 1e-3,
         "max_weight": 10, "min_coeff": 1e-5, "floor": -1},
        # The same family on a small dense lattice (2-word keys, over a million
        # terms): merging dominates.
        {"name": "kicked_6x6", "kind": "kicked", "rows": 6, "cols": 6, "steps": 8, "theta": 0.6, "p": 1e-3,
         "max_weight": 10, "min_coeff": 1e-5, "floor": -1},
        # A wide register (180 qubits, 8-word keys).
        {"name": "kicked_12x15", "kind": "kicked", "rows": 12, "cols": 15, "steps": 8, "theta": 0.6, "p": 1e-3,
         "max_weight": 10, "min_coeff": 1e-5, "floor": -1},
        # A TermBudget floor beside the coefficient cut: truncation is off
        # while fewer terms than the floor are live.
        {"name": "kicked_floor", "kind": "kicked", "rows": 5, "cols": 7, "steps": 6, "theta": 0.6, "p": 2e-3,
         "max_weight": -1, "min_coeff": 1e-3, "floor": 20000},
        # Fermionic circuits: 24 sites, 15M terms.
        {"name": "givens_24", "kind": "givens", "n": 24, "reps": 3, "max_weight": 8, "min_coeff": 1e-6},
        # The largest: 32 sites, 99M terms.
        {"name": "givens_32", "kind": "givens", "n": 32, "reps": 4, "max_weight": 8, "min_coeff": 1e-6},
        # Training: value and gradient of a 50-qubit ansatz, 1,200 angles.
        {"name": "ansatz_50q", "kind": "ansatz", "n": 50, "layers": 12, "sigma": 0.1, "max_weight": 8,
         "min_coeff": 1e-5},
        # An extrapolation sweep: 16 uneven instances in one batch.
        {"name": "sweep_16", "kind": "sweep", "instances": 16, "n_lo": 40, "n_hi": 100, "steps_lo": 8, "steps_hi": 20},
        # A large observable (60,000 raw terms with repeated keys) through the
        # engine's C ABI, its final terms read back in key order.
        {"name": "terms_100q", "kind": "terms", "n": 100, "raw": 60000, "distinct": 9000, "gates": 40,
         "max_weight": 5, "min_coeff": 1e-4},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _log_int(rng, lo, hi):
    return int(min(hi, max(lo, round(_log_uniform(rng, lo, hi)))))


def draw(rng):
    kind = rng.choice(["register", "tfim", "kicked", "kicked", "floor", "givens", "givens", "ansatz", "sweep", "terms"])
    if kind == "register":
        return {"kind": kind, "n": rng.randint(3, 12), "gates": _log_int(rng, 10, 400), "max_weight": rng.randint(3, 6),
                "min_coeff": _log_uniform(rng, 1e-5, 1e-3), "damping": rng.choice([0.0, 0.003, 0.01])}
    if kind == "tfim":
        return {"kind": kind, "n": _log_int(rng, 6, 60), "steps": rng.randint(2, 12), "max_weight": rng.randint(6, 9),
                "min_coeff": _log_uniform(rng, 5e-5, 1e-3)}
    if kind == "kicked":
        return {"kind": kind, "rows": rng.randint(3, 13), "cols": rng.randint(4, 15), "steps": rng.randint(3, 14),
                "theta": rng.uniform(0.2, 1.0), "p": rng.choice([0.0005, 0.001, 0.0015, 0.002]),
                "max_weight": rng.randint(7, 12), "min_coeff": _log_uniform(rng, 1e-5, 1e-3), "floor": -1}
    if kind == "floor":
        return {"kind": "kicked", "rows": rng.randint(3, 8), "cols": rng.randint(4, 10), "steps": rng.randint(3, 6),
                "theta": rng.uniform(0.3, 0.8), "p": rng.choice([0.001, 0.002]), "max_weight": -1,
                "min_coeff": _log_uniform(rng, 5e-4, 3e-3), "floor": _log_int(rng, 1000, 30000)}
    if kind == "givens":
        n = _log_int(rng, 7, 40)
        return {"kind": kind, "n": n, "reps": rng.randint(2, 3), "max_weight": rng.randint(6, 8),
                "min_coeff": _log_uniform(rng, 1e-6, 1e-4)}
    if kind == "ansatz":
        return {"kind": kind, "n": _log_int(rng, 5, 50), "layers": rng.randint(2, 10), "sigma": rng.uniform(0.05, 0.15),
                "max_weight": rng.randint(6, 8), "min_coeff": _log_uniform(rng, 1e-5, 1e-3)}
    if kind == "sweep":
        lo = rng.randint(12, 60)
        return {"kind": kind, "instances": _log_int(rng, 2, 32), "n_lo": lo, "n_hi": rng.randint(lo, 100),
                "steps_lo": 4, "steps_hi": rng.randint(5, 12)}
    raw = _log_int(rng, 500, 60000)
    return {"kind": kind, "n": _log_int(rng, 10, 130), "raw": raw, "distinct": max(50, raw // rng.randint(2, 9)),
            "gates": _log_int(rng, 10, 60), "max_weight": rng.randint(4, 5), "min_coeff": _log_uniform(rng, 1e-4, 1e-2)}


# ------------------------------------------------------------------ inputs
def _string(rng, n, k):
    """A random Pauli string on k of n qubits: (x, z)."""
    x = z = 0
    for q in rng.choice(n, size=k, replace=False):
        t = int(rng.integers(1, 4))
        x |= (t & 1) << int(q)
        z |= (t >> 1) << int(q)
    return x, z


def _random_layers(rng, n, gates, size):
    rots = []
    for _ in range(gates):
        x, z = _string(rng, n, int(rng.integers(1, min(n, 3) + 1)))
        rots.append(PauliRotation(PauliString(x, z, n), float(rng.uniform(-1.2, 1.2))))
    return [rots[i:i + size] for i in range(0, gates, size)]


def _jittered_kicked(rows, cols, steps, theta, p, max_weight, min_coeff, site, rng):
    """workloads.kicked_ising with every RX angle within 1% of theta."""
    wl = workloads.kicked_ising(rows, cols, steps, theta, p, max_weight, min_coeff, site=site)
    for layer in wl.circuit.layers:
        for r in layer:
            if r.angle == theta:
                r.angle = theta * (1.0 + 0.01 * float(rng.uniform(-1.0, 1.0)))
    return wl


def _problems(case, seed):
    """The case's propagations: (workload, TermBudget floor or None)."""
    kind = case["kind"]
    rng = np.random.default_rng([seed, 71])
    if kind == "register":
        n = case["n"]
        obs = PauliTermSum()
        obs.add(PauliString(0, 1, n), 1.0)
        circ = PauliCircuit(_random_layers(rng, n, case["gates"], 1))
        return [(workloads.Workload("register", 0, n, obs, circ, case["max_weight"], case["min_coeff"],
                                    case["damping"] or None, 0), None)]
    if kind == "tfim":
        return [(workloads.tfim_chain(case["n"], case["steps"], seed, case["max_weight"], case["min_coeff"]), None)]
    if kind == "kicked":
        wl = _jittered_kicked(case["rows"], case["cols"], case["steps"], case["theta"], case["p"],
                              None if case["max_weight"] < 0 else case["max_weight"], case["min_coeff"], None, rng)
        return [(wl, None if case["floor"] < 0 else case["floor"])]
    if kind == "givens":
        return [(workloads.majorana_givens(case["n"], case["reps"], seed, case["max_weight"], case["min_coeff"]), None)]
    if kind == "ansatz":
        return [(workloads.hardware_efficient(case["n"], case["layers"], seed, case["sigma"], case["max_weight"],
                                              case["min_coeff"]), None)]
    if kind == "sweep":
        # the instances' sizes belong to the case, their angles to the seed
        out = []
        for wl in workloads.kicked_ising_batch(case["instances"], 0, (case["n_lo"], case["n_hi"]),
                                               (case["steps_lo"], case["steps_hi"])):
            rows, cols = workloads.most_square_grid(wl.n_units)
            out.append((_jittered_kicked(rows, cols, wl.meta["steps"], wl.meta["theta"], wl.meta["p"], wl.max_weight,
                                         wl.min_coeff, wl.meta["site"], rng), None))
        return out
    raise ValueError(kind)


def _interleave(x, z, n):
    key = 0
    for q in range(n):
        key |= (x >> q & 1) << (2 * q) | (z >> q & 1) << (2 * q + 1)
    return key


def _terms_arrays(case, seed):
    """The C-ABI arrays of a 'terms' case."""
    rng = np.random.default_rng([seed, 72])
    n = case["n"]
    W = _native.words_for_units(n)
    circ = PauliCircuit(_random_layers(rng, n, case["gates"], 4))
    gw, ga, off = heisenberg_gates(circ, W, lambda g: g.key())
    d = case["distinct"]
    place = np.argsort(rng.random((d, n)), axis=1)[:, :min(4, n)]  # up to 4 distinct qubits a key
    kind = rng.integers(1, 4, size=place.shape).astype(np.uint64)
    kind *= np.arange(place.shape[1]) < rng.integers(1, place.shape[1] + 1, size=(d, 1))
    keys = np.zeros((d, W), dtype=np.uint64)
    for j in range(place.shape[1]):
        np.bitwise_or.at(keys, (np.arange(d), place[:, j] // 32), kind[:, j] << (2 * (place[:, j] % 32)).astype(np.uint64))
    pick = rng.integers(0, d, size=case["raw"])
    coeffs = rng.normal(size=case["raw"]) * 10.0 ** rng.integers(-2, 1, size=case["raw"])
    return np.ascontiguousarray(keys[pick]), coeffs, gw, ga, off, state_words(5 % (1 << min(n, 60)), n), W


def _propagator(wl, floor):
    cls = pq.PauliPropagator if wl.basis == 0 else pq.MajoranaPropagator
    trunc = wl.truncation()
    if floor is not None:
        trunc.append(pq.TermBudget(floor))
    return cls(noise=wl.noise(), truncation=trunc)


_ROOM = 1 << 19


def prepare(case, seed):
    if case["kind"] == "terms":
        obs_keys, obs_coeffs, gw, ga, off, diag, W = _terms_arrays(case, seed)
        cfg = _native.RunConfig()
        cfg.basis_kind, cfg.n_units = 0, case["n"]
        cfg.max_weight, cfg.has_min_coeff, cfg.min_coeff, cfg.min_terms = case["max_weight"], 1, case["min_coeff"], -1
        cfg.want_terms = 2
        # the caller's own arrays for the final terms, larger than any result
        return {"kind": "terms", "engine": _native.engine(0), "words": W, "keys": np.zeros((_ROOM, W), dtype=np.uint64),
                "coeffs": np.zeros(_ROOM), "args": (cfg, obs_keys, obs_coeffs, gw, ga, off, diag)}
    probs = _problems(case, seed)
    if case["kind"] == "sweep":
        return {"kind": "sweep", "jobs": [(_propagator(wl, fl), wl.observable, wl.circuit, wl.initial_state)
                                          for wl, fl in probs]}
    wl, floor = probs[0]
    prop = _propagator(wl, floor)
    if case["kind"] == "ansatz":
        spec = ParametrizedExpectation(prop, wl.observable, wl.circuit, wl.meta["param_index"],
                                       initial_state=wl.initial_state)
        return {"kind": "ansatz", "spec": spec, "theta": wl.meta["theta"]}
    return {"kind": "one", "prop": prop, "args": (wl.observable, wl.circuit, wl.initial_state)}


def _outputs(r):
    return {"value": r.expectation_value, "n_terms": np.asarray(r.n_terms, dtype=np.int64), "below": r.terms_below_cutoff}


def run(state):
    kind = state["kind"]
    if kind == "one":
        return _outputs(state["prop"].expectation_value(*state["args"]))
    if kind == "sweep":
        res = expectation_values(state["jobs"])
        return {"values": np.array([r.expectation_value for r in res]),
                "n_terms": np.concatenate([np.asarray(r.n_terms, dtype=np.int64) for r in res]),
                "below": np.array([r.terms_below_cutoff for r in res])}
    if kind == "ansatz":
        value, grad = state["spec"].value_and_grad(state["theta"])
        return {"value": value, "grad": grad}
    res, n_terms = state["engine"].run(*state["args"])
    keys, coeffs = state["engine"].terms(state["words"])
    state["keys"][:len(coeffs)] = keys
    state["coeffs"][:len(coeffs)] = coeffs
    return {"value": res.expectation_value, "n_terms": n_terms, "keys": state["keys"], "coeffs": state["coeffs"]}


def work(case):
    """Inputs read once (terms, rotations) and results written once (live
    counts, gradient, terms); two products and a sum per rotation."""
    kind = case["kind"]
    if kind == "sweep":
        n = (case["n_lo"] + case["n_hi"]) // 2
        units, gates, obs = n, case["instances"] * 3 * n * ((case["steps_lo"] + case["steps_hi"]) // 2), case["instances"]
    elif kind == "kicked":
        r, c = case["rows"], case["cols"]
        units, gates, obs = r * c, case["steps"] * (3 * r * c - r - c), 1
    elif kind == "tfim":
        units, gates, obs = case["n"], case["steps"] * (2 * case["n"] - 1), 1
    elif kind == "givens":
        units, obs = case["n"], case["n"]
        gates = case["reps"] * (2 * (case["n"] - 1) + 3 * (3 * case["n"] - 6))
    elif kind == "ansatz":
        units, obs = case["n"], case["n"] - 1
        gates = case["layers"] * (2 * case["n"] + 3 * (case["n"] - 1))
    else:
        units, gates, obs = case["n"], case["gates"], case.get("raw", 1)
    row = 8 * _native_words(units) + 8
    out = 8 * gates + (case["distinct"] * row if kind == "terms" else 0)
    return {"bytes": obs * row + gates * row + out, "flops": 3 * gates}


def _native_words(units):
    w = 1
    while 32 * w < units:
        w *= 2
    return w


# ------------------------------------------------- plain numpy restatement
_EVEN = np.uint64(0x5555555555555555)
_ONE = np.uint64(1)
_U = np.uint64


def _popc(a):
    return np.bitwise_count(a).astype(np.int64)


def _weights(k, basis, n):
    """Pauli weight, or the Jordan-Wigner weight of a Majorana monomial."""
    if basis == 0:
        return sum(_popc((k[:, w] | (k[:, w] >> _ONE)) & _EVEN) for w in range(k.shape[1]))
    single = (k ^ (k >> _ONE)) & _EVEN
    odd = sum(_popc(single[:, w]) for w in range(k.shape[1])) & 1
    out = np.zeros(len(k), dtype=np.int64)
    below = np.zeros(len(k), dtype=_U)  # EVEN where the singles of lower words are odd
    for w in range(k.shape[1]):
        sites = min(32, max(0, n - 32 * w))
        live = _U((1 << (2 * sites)) - 1) & _EVEN
        p = single[:, w].copy()
        for s in (2, 4, 8, 16, 32):
            p ^= p << _U(s)
        p ^= below
        below = np.where((p >> _U(62)) & _ONE, _EVEN, _U(0))
        par = np.where(odd, p ^ _EVEN, p) & live
        out += _popc((single[:, w] | ((k[:, w] | (k[:, w] >> _ONE)) & _EVEN ^ par)) & live)
    return out


def _phase(g, k, basis):
    """Exponent p of G K = i^p (G xor K), per row."""
    W = k.shape[1]
    if basis == 0:
        p = np.zeros(len(k), dtype=np.int64)
        for w in range(W):
            o = k[:, w] ^ g[w]
            p += _popc(g[w] & (g[w] >> _ONE) & _EVEN) + _popc(k[:, w] & (k[:, w] >> _ONE) & _EVEN)
            p += 2 * _popc((g[w] >> _ONE) & k[:, w] & _EVEN) - _popc(o & (o >> _ONE) & _EVEN)
        return p & 3
    herm = lambda n: ((n & 3) >= 2).astype(np.int64)  # noqa: E731
    lk = np.zeros(len(k), dtype=np.int64)
    lo, swaps, lg, above = lk.copy(), lk.copy(), 0, 0
    for w in reversed(range(W)):
        s = int(g[w]) >> 1
        for sh in (1, 2, 4, 8, 16, 32):
            s ^= s >> sh
        pk = _popc(k[:, w])
        lk += pk
        lo += _popc(k[:, w] ^ g[w])
        swaps ^= (_popc(k[:, w] & _U(s)) & 1) ^ (pk & above)
        lg += int(g[w]).bit_count()
        above ^= int(g[w]).bit_count() & 1
    return (herm(np.array(lg)) + herm(lk) - herm(lo) + 2 * (swaps & 1)) & 3


def _anti(g, k, basis):
    acc = np.zeros(len(k), dtype=_U)
    for w in range(k.shape[1]):
        f = int(g[w])
        if basis == 0:
            f = (f & int(_EVEN)) << 1 | (f >> 1) & int(_EVEN)
        if f:
            acc ^= k[:, w] & _U(f)
    par = _popc(acc) & 1
    if basis == 1 and sum(int(v).bit_count() for v in g) & 1:
        par = par ^ (sum(_popc(k[:, w]) for w in range(k.shape[1])) & 1)
    return par.astype(bool)


def _mix(k):
    """A 64-bit hash per key, for finding partners."""
    h = np.zeros(len(k), dtype=_U)
    for w in range(k.shape[1]):
        h = (h ^ k[:, w]) * _U(0x9E3779B97F4A7C15)
        h ^= h >> _U(29)
        h *= _U(0xBF58476D1CE4E5B9)
        h ^= h >> _U(32)
    return h


_VISITS = 1.7e9  # row visits (3 each, 60 more where a row branches) of about 15 seconds


def _propagate(keys, coeffs, gates, angles, offsets, basis, n, wcut, ccut, floor, damping, spend, grad_of=None, state=0):
    """Gate by gate: pair, branch, truncate, damp.  Returns (keys, coeffs,
    n_terms, value, dE/dangle) or None past the visits allowed."""
    first = {}
    rows, vals = [], []
    for k, c in zip(map(bytes, keys), coeffs):  # duplicates add up in input order
        if k in first:
            vals[first[k]] += c
        else:
            first[k] = len(rows)
            rows.append(k)
            vals.append(c)
    K = np.frombuffer(b"".join(rows), dtype=_U).reshape(-1, keys.shape[1]).copy()
    C = np.array(vals, dtype=np.float64)
    n_terms = np.zeros(len(angles), dtype=np.int64)
    tape = []
    frame = []  # Clifford rotations kept out of the term sum (all of them without a weight cut): (generator, sin)
    for layer in range(len(offsets) - 1):
        if damping is not None:
            w = _weights(K, basis, n)
            f = np.array([math.exp(-damping * float(i)) for i in range(n + 1)])[w]
            C = C * f
            if wcut is not None or ccut is not None:
                keep = np.ones(len(C), dtype=bool)
                if wcut is not None:
                    keep &= w <= wcut
                if ccut is not None:
                    keep &= np.abs(C) >= ccut
                K, C = K[keep], C[keep]
            else:
                keep = slice(None)
            tape.append((0, f, keep))
        for gi in range(offsets[layer], offsets[layer + 1]):
            g, sn, cs = gates[gi], math.sin(angles[gi]), math.cos(angles[gi])
            if abs(cs) < 1e-9 and wcut is None:
                frame.append((g, round(sn)))
                n_terms[gi] = len(K)
                continue
            g, sign = _into_frame(g, frame, basis)
            A = np.nonzero(_anti(g, K, basis))[0]
            spend[0] -= 3 * len(K) + 60 * len(A)
            if spend[0] < 0:
                return None
            Q = K[A] ^ g
            s = np.where(_phase(g, K[A], basis) == 1, -sign, sign)
            one_unit = sum(int(v | (v >> _ONE)) & int(_EVEN) for v in g).bit_count() == 1
            if abs(cs) < 1e-9 and basis == 0 and one_unit:  # keeps weights: a relabelling of the terms
                K[A] = Q
                C[A] = C[A] * (s * round(sn))
                tape.append((1, A, s * round(sn)))
                n_terms[gi] = len(K)
                continue
            c = C[A]
            if abs(sn) < 1e-9:
                C[A] = c * cs
                tape.append((2, gi, A, c, s, sn, cs, np.full(len(A), -1), np.zeros(len(A), bool), len(K)))
                n_terms[gi] = len(K)
                continue
            lossless = floor is not None and len(K) < floor
            hk, hq = _mix(K[A]), _mix(Q)
            order = np.argsort(hk)
            at = np.minimum(np.searchsorted(hk, hq, sorter=order), max(0, len(A) - 1))
            j = order[at] if len(A) else at
            found = hk[j] == hq if len(A) else np.zeros(0, bool)
            b = (c * sn) * s
            held = np.zeros(len(A), dtype=bool)
            drop = np.zeros(len(A), dtype=bool)
            if ccut is not None and not lossless:
                held = np.abs(c * sn) < ccut
            if wcut is not None and not lossless:
                drop = ~held & (_weights(Q, basis, n) > wcut)
            emit = ~held & ~drop
            sent = np.where(found, emit | (held & emit[j]), emit) if len(A) else emit
            new = c * cs
            src = np.nonzero(found & sent)[0]
            new[j[src]] += b[src]
            C[A] = new
            lone = np.nonzero(~found & sent)[0]
            to = np.where(found, A[j] if len(A) else A, -1)
            to[lone] = len(K) + np.arange(len(lone))
            tape.append((2, gi, A, c, s, sn, cs, to, sent, len(K)))
            if len(lone):
                K = np.concatenate([K, Q[lone]])
                C = np.concatenate([C, b[lone]])
            n_terms[gi] = len(K)
        if grad_of is None:
            tape.clear()
    for g, sn in frame:
        A = np.nonzero(_anti(g, K, basis))[0]
        C[A] *= np.where(_phase(g, K[A], basis) == 1, -sn, sn)
        K[A] ^= g
    tr = _traces(K, basis, n, state)
    value = math.fsum((C * tr).tolist())
    grad = None
    if grad_of is not None:
        grad = np.zeros(len(angles))
        lam = tr.copy()
        for step in reversed(tape):
            if step[0] == 0:
                full = np.zeros(len(step[1]))
                full[step[2]] = lam
                lam = full * step[1]
            elif step[0] == 1:
                lam[step[1]] *= step[2]
            else:
                _, gi, A, c, s, sn, cs, to, sent, n_in = step
                t = np.nonzero(sent)[0]
                grad[gi] = -sn * float(c @ lam[A]) + cs * float((s[t] * c[t]) @ lam[to[t]])
                back = cs * lam[A]
                back[t] += sn * s[t] * lam[to[t]]
                lam[A] = back
                lam = lam[:n_in]
    return K, C, n_terms, value, grad



def _into_frame(g, frame, basis):
    """The generator and sign that act on the stored terms as g acts on the
    true ones: the deferred rotations undone, last one first."""
    k, sign = g.reshape(1, -1).copy(), 1.0
    for f, sn in reversed(frame):
        if _anti(f, k, basis)[0]:
            sign *= sn if _phase(f, k, basis)[0] == 1 else -sn
            k = k ^ f
    return k[0], sign


def _traces(K, basis, n, state):
    W = K.shape[1]
    bits = np.zeros(W, dtype=_U)
    for u in range(n):
        if int(state) >> u & 1:
            pos = 2 * u + (1 if basis == 0 else 0)
            bits[pos // 64] |= _U(1 << (pos % 64))
    bad = np.zeros(len(K), dtype=bool)
    par = np.zeros(len(K), dtype=np.int64)
    pairs = par.copy()
    for w in range(W):
        if basis == 0:
            bad |= (K[:, w] & _EVEN) != 0
            par += _popc(K[:, w] & bits[w])
        else:
            bad |= ((K[:, w] ^ (K[:, w] >> _ONE)) & _EVEN) != 0
            pr = K[:, w] & _EVEN
            pairs += _popc(pr)
            par += _popc(pr & ~bits[w])
    sign = np.where(((par & 1) ^ ((pairs >> 1) & 1)) == 1, -1.0, 1.0)
    return np.where(bad, 0.0, sign)


def exact(case, seed):
    spend = [_VISITS]
    if case["kind"] == "terms":
        ok, oc, gw, ga, off, diag, W = _terms_arrays(case, seed)
        w = _weights(ok, 0, case["n"])
        keep = (w <= case["max_weight"]) & (np.abs(oc) >= case["min_coeff"])
        got = _propagate(ok[keep], oc[keep], gw, ga, off, 0, case["n"], case["max_weight"], case["min_coeff"], None,
                         None, spend, state=5 % (1 << min(case["n"], 60)))
        if got is None:
            return None
        coeffs = np.zeros(_ROOM)
        coeffs[:len(got[1])] = got[1][np.lexsort(got[0].T)]
        return {"value": got[3], "n_terms": None, "keys": None, "coeffs": coeffs}
    out = []
    for wl, floor in _problems(case, seed):
        W = _native_words(wl.n_units)
        ok, oc = wl.observable.to_arrays(W)
        gw, ga, off = heisenberg_gates(wl.circuit, W, lambda g: g.key())
        keep = np.ones(len(oc), dtype=bool)
        if wl.max_weight is not None:
            keep &= _weights(ok, wl.basis, wl.n_units) <= wl.max_weight
        if wl.min_coeff is not None:
            keep &= np.abs(oc) >= wl.min_coeff
        got = _propagate(ok[keep], oc[keep], gw, ga, off, wl.basis, wl.n_units, wl.max_weight, wl.min_coeff, floor,
                         wl.noise_damping, spend, grad_of=case["kind"] == "ansatz" or None, state=wl.initial_state)
        if got is None:
            return None
        if case["kind"] == "ansatz":
            idx = np.asarray(wl.meta["param_index"])[_heisenberg_index(wl.circuit)]
            grad = np.zeros(len(wl.meta["theta"]))
            np.add.at(grad, idx[idx >= 0], got[4][idx >= 0])
            return {"value": got[3], "grad": grad}
        out.append({"value": got[3], "n_terms": None, "below": None})
    if case["kind"] == "sweep":
        return {"values": np.array([o["value"] for o in out]), "n_terms": None, "below": None}
    return out[0]


def _heisenberg_index(circuit):
    starts, k = [], 0
    for layer in circuit.layers:
        starts.append((k, len(layer)))
        k += len(layer)
    return np.array([s + i for s, m in reversed(starts) for i in reversed(range(m))], dtype=np.int64)
