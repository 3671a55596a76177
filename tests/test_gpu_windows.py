"""Windows of the binned sweep (propaq_b200/csrc/pq_host.cu, plan_windows)
against the oracle: live count after every rotation, branching rows, term set,
every coefficient bit for bit, expectation value.

* Rotations by pi across a layer of rotations on disjoint qubits: they share
  its window and need not commute with it, so a row born inside the window may
  anticommute with one although no row entering it does.
* Live sets that double with every rotation, so that buffers of the first size
  are asked for very many bins.
* Groups that the 32-bit group hash cannot tell apart and that one block cannot
  hold together: the run takes the row sweep.
* Windows that multiply their rows by up to 2^11, so that the next window's
  bins, laid out before, hold many times too few.
* Registers so small that their live set fills the key space, and circuits so
  short that one block certainly runs them."""

from __future__ import annotations

import math

import numpy as np
import pytest
from harness import (assert_terms_equal, expectation_close, from_circuit, make_cfg, run_gpu, run_gpu_batch, run_oracle)

from propaq_b200 import _native
from propaq_b200.circuits import MajoranaCircuit, MajoranaRotation, PauliCircuit, PauliRotation
from propaq_b200.datatypes import MajoranaMonomial, MajoranaTermSum, PauliString, PauliTermSum


def check(g, o):
    assert np.array_equal(g.n_terms, o.n_terms), "live counts per gate differ"
    assert_terms_equal(g.keys, g.coeffs, o.keys, o.coeffs)
    assert g.terms_below_cutoff == o.terms_below_cutoff
    assert expectation_close(g.expectation, o)[0]


def echo(n, cut):
    """Z on qubit 0 under RX(0.3), RZ(pi), RX(0.3) on every qubit: the second
    layer undoes the first, <Z> = 1."""
    x = [PauliRotation(PauliString(1 << q, 0, n), 0.3) for q in range(n)]
    z = [PauliRotation(PauliString(0, 1 << q, n), math.pi) for q in range(n)]
    return from_circuit(0, n, PauliTermSum({PauliString(0, 1, n): 1.0}), PauliCircuit([x, z, x]), 0, max_weight=cut)


def pulses(seed, n, n_terms, cut, min_coeff):
    """Layers of one-qubit rotations on every qubit, with rotations by multiples
    of pi about random one- and two-qubit Paulis between and after them."""
    rng = np.random.default_rng(seed)

    def pauli(k):
        x = z = 0
        for q in rng.choice(n, size=k, replace=False):
            t = int(rng.integers(1, 4))
            x |= (t & 1) << int(q)
            z |= (t >> 1) << int(q)
        return PauliString(x, z, n)

    layers = []
    for _ in range(3):
        layer = []
        for q in range(n):
            t = int(rng.integers(1, 4))
            layer.append(PauliRotation(PauliString((t & 1) << q, (t >> 1) << q, n), float(rng.uniform(0.1, 1.4))))
            if rng.random() < 0.3:
                layer.append(PauliRotation(pauli(int(rng.integers(1, 3))), math.pi * int(rng.integers(1, 4))))
        layers.append(layer[:126])
    obs = {}
    while len(obs) < n_terms:
        obs[pauli(int(rng.integers(1, 5)))] = float(rng.normal())
    return from_circuit(0, n, PauliTermSum(obs), PauliCircuit(layers), 5, max_weight=cut, min_coeff=min_coeff)


@pytest.mark.gpu
@pytest.mark.parametrize("n,cut", [(20, 8), (20, 11), (50, 11), (100, 11), (100, 8), (180, 10)])
def test_echo_across_a_disjoint_window(gpu_engine, oracle, n, cut):
    p = echo(n, cut)
    g = run_gpu(gpu_engine, p)
    check(g, run_oracle(oracle, p))
    assert abs(g.expectation - 1.0) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("n,cut", [(20, 11), (50, 10), (100, 11), (180, 10)])
@pytest.mark.parametrize("n_terms", [1, 40, 500])
def test_pulses_in_disjoint_windows(gpu_engine, oracle, n, cut, n_terms):
    # one term: a warp alone; 40: a block; 500: bins of warps and of blocks
    p = pulses(n + n_terms, n, n_terms, cut, 1e-3)
    check(run_gpu(gpu_engine, p), run_oracle(oracle, p))


@pytest.mark.gpu
def test_pulses_in_a_batch(gpu_engine, oracle):
    probs = [echo(20, 9), pulses(1, 30, 4, 10, 1e-3), pulses(2, 60, 60, 9, 1e-2), echo(100, 11)]
    for p, g in zip(probs, run_gpu_batch(gpu_engine, probs)):
        check(g, run_oracle(oracle, p))


@pytest.mark.gpu
@pytest.mark.parametrize("n,width", [(24, 200), (25, 90), (26, 26)], ids=["W8", "W4", "W1"])
def test_doubling_past_every_buffer(n, width):
    # Z on n qubits under RX on each of them: 2^n rows, <0|..|0> = prod cos.  A
    # fresh engine, so every buffer starts at its first size.
    rng = np.random.default_rng(n)
    angles = rng.uniform(0.3, 1.2, n)
    x = [PauliRotation(PauliString(1 << q, 0, width), float(angles[q])) for q in range(n)]
    zz = [PauliRotation(PauliString(0, 3 << q, width), 0.4) for q in (0, 2)]
    p = from_circuit(0, width, PauliTermSum({PauliString(0, (1 << n) - 1, width): 1.0}), PauliCircuit([zz, x]), 0)
    g = run_gpu(_native.Engine(0), p, want_terms=False)
    # every row has Y or Z on each qubit; of the four pairs a ZZ rotation
    # branches two, into two new ones
    assert g.n_terms.tolist() == [2 << q for q in range(n)] + [3 << (n - 1), 9 << (n - 2)]
    assert abs(g.expectation - float(np.prod(np.cos(angles)))) < 1e-12


# ------------------------------------------- groups that cannot be told apart
def hash_kernel(lowest_bit):
    """A nonzero one-word key on bits >= lowest_bit whose linear hash (lin_table
    of pq_host.cu) is 0: keys that differ by it share every group hash."""
    mask = (1 << 64) - 1
    x, bits = 0x1234567890ABCDEF, []
    for _ in range(64):
        x = (x + 0x9E3779B97F4A7C15) & mask
        z = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        bits.append(((z ^ (z >> 31)) >> 16) & 0xFFFFFFFF)
    rows = {}
    for b in range(lowest_bit, 64):
        h, c = bits[b], 1 << b
        while h and h.bit_length() in rows:
            hh, cc = rows[h.bit_length()]
            h, c = h ^ hh, c ^ cc
        if not h:
            return c
        rows[h.bit_length()] = (h, c)
    raise AssertionError("the hash is injective on these bits")


def colliding_groups(n):
    """Two terms whose keys differ by a kernel vector of the hash, each grown
    to 2^11 rows by RX on qubits 0..10: one unsplittable bin of 4,096 rows."""
    low = 3  # X and Z bits of qubits 0..10 stay clear of the vector
    d = hash_kernel(22)
    z11 = sum(1 << q for q in range(11))
    dx, dz = (sum(((d >> (2 * q + b)) & 1) << q for q in range(11, 32)) for b in (0, 1))
    obs = PauliTermSum({PauliString(0, z11, n): 1.0, PauliString(dx, dz | z11, n): 0.5, PauliString(0, low, n): 0.25})
    rx = [PauliRotation(PauliString(1 << q, 0, n), 0.2 + 0.05 * q) for q in range(11)]
    rzz = [PauliRotation(PauliString(0, 3 << q, n), 0.3) for q in range(4)]
    p = from_circuit(0, n, obs, PauliCircuit([rzz, rx]), 0)
    k0, k1 = (int(k[0]) for k in p.obs_keys[np.argsort(-np.abs(p.obs_coeffs))][:2])
    assert k0 ^ k1 == d
    return p


@pytest.mark.gpu
@pytest.mark.parametrize("n", [32, 120], ids=["W1", "W4"])
def test_bins_that_cannot_be_split(gpu_engine, oracle, n):
    p = colliding_groups(n)
    o = run_oracle(oracle, p)
    check(run_gpu(gpu_engine, p), o)
    for g in run_gpu_batch(gpu_engine, [p, p]):
        check(g, o)


# -------------------------------------------------- windows that multiply rows
@pytest.mark.gpu
@pytest.mark.parametrize("k,n,width,pairs", [(0, 22, 22, ()), (0, 22, 120, ()), (0, 22, 22, (0, 2)),
                                             (0, 22, 120, (0, 2)), (3, 22, 30, (0, 2)), (4, 22, 120, (0, 2))],
                         ids=["W1-2^22", "W4-2^22", "W1-2^22-ZZ", "W4-2^22-ZZ", "W1-2^25-ZZ", "W4-2^26-ZZ"])
def test_windows_that_multiply_their_rows(k, n, width, pairs):
    # 2^k Z strings under RX on n qubits, then ZZ rotations, against the row
    # sweep (a knob at its default takes it): the same counts and value, and in
    # a time of the same order.  The first two take 0.7 and 0.9 ms on both
    # sweeps (4.1 and 4.6 on the binned one while a pair of groups could send a
    # block's bins deep); the last two 8.7 and 20 ms on the row sweep and 8.0
    # and 31 on the binned one (73 and 3,040 before rows were dealt again).
    rng = np.random.default_rng(k)
    angles = rng.uniform(0.3, 1.2, n)
    x = [PauliRotation(PauliString(1 << q, 0, width), float(angles[q])) for q in range(n)]
    zz = [PauliRotation(PauliString(0, 3 << q, width), 0.4) for q in pairs]
    obs = PauliTermSum({PauliString(0, ((1 << n) - 1) | i << n, width): float(rng.normal()) for i in range(1 << k)})
    p = from_circuit(0, width, obs, PauliCircuit([zz, x]), 0)
    engine = _native.Engine(0)
    cfg, keep = make_cfg(p, want_terms=False)
    runs = []
    for knob in (0, 2):
        cfg.fuse_max = knob  # the first run grows the buffers; the fastest of the others counts
        several = [engine.run(cfg, p.obs_keys, p.obs_coeffs, p.gate_keys, p.angles, p.offsets, p.diag) for _ in range(4)]
        runs.append(min(several[1:], key=lambda r: r[0].device_ms))
    (binned, nb), (row, nr) = runs
    assert np.array_equal(nb, nr) and int(nb[-1]) == 3 ** len(pairs) << (k + n - len(pairs))
    for f in ("n_final", "peak_terms", "sum_anti", "sum_children", "sum_rows_gate"):
        assert getattr(binned, f) == getattr(row, f), f
    want = float(np.sum(p.obs_coeffs)) * float(np.prod(np.cos(angles)))
    for r in (binned, row):
        assert abs(r.expectation_value - want) <= 1e-12 * float(np.sum(np.abs(p.obs_coeffs)))
    assert binned.device_ms < 3.0 * row.device_ms


# --------------------------------------------------------- small registers
def full_majorana(sites, n_gates):
    rng = np.random.default_rng(sites)
    m = 2 * sites
    rots = []
    for _ in range(n_gates):
        modes = rng.choice(m, size=int(rng.integers(1, 5)), replace=False)
        rots.append(MajoranaRotation(MajoranaMonomial(sum(1 << int(v) for v in modes), m, False),
                                     float(rng.uniform(-1, 1))))
    obs = MajoranaTermSum()
    obs.add(MajoranaMonomial(3, m), 1.0)
    return from_circuit(1, sites, obs, MajoranaCircuit([rots]), 5)


def full_pauli(n, n_gates):
    rng = np.random.default_rng(n)
    rots = []
    for _ in range(n_gates):
        x = z = 0
        for q in rng.choice(n, size=min(n, int(rng.integers(1, 4))), replace=False):
            t = int(rng.integers(1, 4))
            x |= (t & 1) << int(q)
            z |= (t >> 1) << int(q)
        rots.append(PauliRotation(PauliString(x, z, n), float(rng.uniform(-1.2, 1.2))))
    return from_circuit(0, n, PauliTermSum({PauliString(0, 1, n): 1.0}), PauliCircuit([rots]), 3)


@pytest.mark.gpu
@pytest.mark.parametrize("make", [lambda: full_majorana(7, 90), lambda: full_majorana(9, 130), lambda: full_pauli(5, 60),
                                  lambda: full_pauli(6, 60), lambda: full_pauli(9, 90)],
                         ids=["7 sites", "9 sites", "5 qubits", "6 qubits", "9 qubits"])
def test_live_sets_that_fill_the_key_space(gpu_engine, oracle, make):
    p = make()
    g = run_gpu(gpu_engine, p)
    check(g, run_oracle(oracle, p))
    assert g.n_final > (1 << (2 * p.n_units)) // 4
    # and not slower than a pass per rotation by much (9 sites: 0.7-1.2 ms
    # against 1.4-2.2; 2.2-7.7 with windows as long as on wide registers)
    cfg, keep = make_cfg(p, want_terms=False)
    best = []
    for knob in (0, 2):
        cfg.fuse_max = knob
        best.append(min(gpu_engine.run(cfg, p.obs_keys, p.obs_coeffs, p.gate_keys, p.angles, p.offsets, p.diag)[0].device_ms
                        for _ in range(4)))
    assert best[0] < 1.5 * best[1]


@pytest.mark.gpu
@pytest.mark.parametrize("n_terms,n_gates", [(1, 0), (1, 1), (1, 11), (1, 12), (511, 2), (512, 2), (513, 2), (1024, 1),
                                             (1025, 1), (1025, 0)])
def test_short_circuits(gpu_engine, oracle, n_terms, n_gates):
    # every rotation doubles every row: on either side of what one block runs
    n = 24
    rng = np.random.default_rng(n_terms)
    x = [PauliRotation(PauliString(1 << q, 0, n), float(rng.uniform(0.3, 1.2))) for q in range(n_gates)]
    obs = PauliTermSum({PauliString(0, ((1 << 12) - 1) | i << 12, n): float(rng.normal()) for i in range(n_terms)})
    p = from_circuit(0, n, obs, PauliCircuit([x] if x else []), 0)
    g = run_gpu(gpu_engine, p)
    check(g, run_oracle(oracle, p))
    assert g.n_final == n_terms << n_gates
    alone = n_gates == 0 or n_terms << (n_gates - 1) <= 1024
    if alone:
        assert g.res.sweep_launches == 1
