"""The binned sweep (propaq_b200/csrc/pq_bins.cuh) where it can go wrong, each
case against the oracle: live count after every rotation, term set, every
coefficient bit for bit, terms below the cutoff, expectation value.

* observables around the rows one warp and one block hold (solo runs, and the
  hand-over to the grid) for 1-, 2-, 4- and 8-word keys;
* live sets of a few rows per warp, and on either side of the line between
  bins of warps and bins of blocks;
* groups as large as a window's span allows (dense cosets), and more rows than
  the bins hold, so that bins are split;
* buffers that grow mid-run on a fresh engine, final rows included;
* the same in a batch, whose instances share those buffers;
* weight cuts around the limit of disjoint windows, phase-only rotations,
  layered noise tables, empty layers, odd Majorana generators."""

import math

import numpy as np
import pytest
from harness import (Problem, assert_terms_equal, expectation_close, from_circuit, from_workload,
                     random_pauli_problem, run_gpu, run_gpu_batch, run_oracle)

from propaq_b200 import _native, workloads
from propaq_b200.circuits import MajoranaCircuit, MajoranaRotation, PauliCircuit, PauliRotation
from propaq_b200.datatypes import MajoranaMonomial, MajoranaTermSum, PauliString, PauliTermSum

pytestmark = pytest.mark.gpu


def check(engine, oracle, p):
    g = run_gpu(engine, p)
    o = run_oracle(oracle, p)
    assert np.array_equal(g.n_terms, o.n_terms), "live counts per gate differ"
    assert_terms_equal(g.keys, g.coeffs, o.keys, o.coeffs)
    assert g.terms_below_cutoff == o.terms_below_cutoff
    assert expectation_close(g.expectation, o)[0]
    return g


def observable(n, n_terms, W, seed):
    """n_terms distinct Pauli keys of weight at most 4."""
    rng = np.random.default_rng(seed)
    keys = set()
    while len(keys) < n_terms:
        k = 0
        for q in rng.choice(n, size=int(rng.integers(1, 5)), replace=False):
            k |= int(rng.integers(1, 4)) << (2 * int(q))
        keys.add(k)
    arr = np.array([[(k >> (64 * w)) & ((1 << 64) - 1) for w in range(W)] for k in sorted(keys)], dtype=np.uint64)
    return arr, rng.normal(size=n_terms)


@pytest.mark.parametrize("n", [24, 60, 120, 250], ids=["W1", "W2", "W4", "W8"])
@pytest.mark.parametrize("n0", [63, 64, 65, 1023, 1024, 1025, 2051, 7171, 40000])
def test_rows_around_one_unit(gpu_engine, oracle, n, n0):
    base = random_pauli_problem(n, n, n_gates=24, max_weight=6, min_coeff=1e-3)
    keys, coeffs = observable(n, n0, base.n_words, n0)
    p = Problem(0, n, base.n_words, keys, coeffs, base.gate_keys, base.angles, base.offsets, base.diag, 6, 1e-3)
    p.noise_table = np.array([math.exp(-0.01 * w) for w in range(n + 1)])
    check(gpu_engine, oracle, p)


@pytest.mark.parametrize("n,width", [(13, 13), (15, 40), (13, 70), (12, 140)], ids=["W1", "W2", "W4", "W8"])
def test_dense_groups(gpu_engine, oracle, n, width):
    # Z on every one of n qubits under X and XX rotations: all 2^n keys of one
    # coset become live, in windows that hold 2^11 (2^10) of them each.
    rng = np.random.default_rng(n)
    x = lambda *qs: PauliString(sum(1 << q for q in qs), 0, width)  # noqa: E731
    layers = [[PauliRotation(x(q), float(rng.uniform(0.3, 1.2))) for q in range(n)],
              [PauliRotation(x(q, (q + 1) % n), float(rng.uniform(0.3, 1.2))) for q in range(n)]]
    obs = PauliTermSum({PauliString(0, (1 << n) - 1, width): 1.0, PauliString(0, 5, width): 0.5})
    g = check(gpu_engine, oracle, from_circuit(0, width, obs, PauliCircuit(layers), 0))
    assert g.n_final > 1 << (n - 1)


@pytest.mark.parametrize("make", [lambda: workloads.kicked_ising(6, 6, 7), lambda: workloads.kicked_ising(4, 4, 6),
                                  lambda: workloads.majorana_givens(18, 3)], ids=["kicked6x6", "kicked4x4", "givens18"])
def test_buffers_grow_on_a_fresh_engine(oracle, make):
    engine = _native.Engine(0)
    p = from_workload(make())
    a = check(engine, oracle, p)
    b = run_gpu(engine, p)  # nothing left to grow
    assert a.res.sweep_launches >= b.res.sweep_launches
    assert np.array_equal(a.keys, b.keys) and np.array_equal(a.coeffs, b.coeffs) and a.expectation == b.expectation


def test_batch_grows_on_a_fresh_engine(oracle):
    # Instances of every width, some ending solo, two outgrowing their buffers
    # (they are run again by themselves), one observable folded on the device.
    engine = _native.Engine(0)
    probs = [from_workload(w) for w in (workloads.kicked_ising(4, 4, 6), workloads.tfim_chain(8, 2),
                                        workloads.kicked_ising(6, 6, 6), workloads.kicked_ising(9, 15, 3),
                                        workloads.kicked_ising(7, 10, 2), workloads.tfim_chain(20, 6))]
    base = random_pauli_problem(3, 20, n_gates=24, max_weight=6, min_coeff=1e-3)
    keys, coeffs = observable(20, 12000, 1, 3)
    probs.append(Problem(0, 20, 1, np.concatenate([keys] * 3), np.concatenate([coeffs, 0.5 * coeffs, coeffs]),
                         base.gate_keys, base.angles, base.offsets, base.diag, 6, 1e-3))
    for _ in range(2):
        for p, b in zip(probs, run_gpu_batch(engine, probs)):
            o = run_oracle(oracle, p)
            assert np.array_equal(b.n_terms, o.n_terms)
            assert_terms_equal(b.keys, b.coeffs, o.keys, o.coeffs)
            assert expectation_close(b.expectation, o)[0]


@pytest.mark.parametrize("shape,cut", [((5, 7), 10), ((5, 7), 11), ((5, 7), 12), ((9, 15), 10), ((9, 15), 11)])
def test_weight_cuts_around_the_disjoint_limit(gpu_engine, oracle, shape, cut):
    check(gpu_engine, oracle, from_workload(workloads.kicked_ising(*shape, 4, 0.7, max_weight=cut, min_coeff=1e-4)))


@pytest.mark.parametrize("n", [10, 45, 90, 200])
def test_phases_layered_noise_and_empty_layers(gpu_engine, oracle, n):
    rng = np.random.default_rng(n)
    layers = []
    for _ in range(10):
        layer = []
        for _ in range(int(rng.integers(0, 9))):
            k = int(rng.integers(1, 4))
            xz = [0, 0]
            for q in rng.choice(min(n, 9), size=k, replace=False):
                t = int(rng.integers(1, 4))
                xz[0] |= (t & 1) << int(q)
                xz[1] |= (t >> 1) << int(q)
            layer.append(PauliRotation(PauliString(*xz, n), math.pi * float(rng.choice([0.13, 1.0, 0.4, 2.0]))))
        layers.append(layer)
    obs = PauliTermSum({PauliString(0, 1, n): 1.0, PauliString(3, 6, n): -0.3})
    for cuts in (dict(max_weight=5, min_coeff=1e-5), dict(min_coeff=1e-4), dict()):
        p = from_circuit(0, n, obs, PauliCircuit(layers), 3, **cuts)
        p.noise_tables_layered = np.exp(-np.outer(np.linspace(0.001, 0.05, len(layers)), np.arange(n + 1)))
        check(gpu_engine, oracle, p)


@pytest.mark.parametrize("sites", [9, 40, 70, 150], ids=["W1", "W2", "W4", "W8"])
def test_odd_majorana_generators(gpu_engine, oracle, sites):
    rng = np.random.default_rng(sites)
    n_modes = 2 * sites
    rots = []
    for _ in range(60):
        modes = rng.choice(n_modes, size=int(rng.integers(1, 5)), replace=False)
        m = sum(1 << int(v) for v in modes)
        rots.append(MajoranaRotation(MajoranaMonomial(m, n_modes, False), float(rng.uniform(-1, 1))))
    obs = MajoranaTermSum()
    for k in (0, sites // 2, sites - 1):
        obs.add(MajoranaMonomial(3 << (2 * k), n_modes), float(rng.normal()))
    layers = [rots[i:i + 7] for i in range(0, len(rots), 7)]
    check(gpu_engine, oracle, from_circuit(1, sites, obs, MajoranaCircuit(layers), 5, max_weight=sites, min_coeff=1e-4))
