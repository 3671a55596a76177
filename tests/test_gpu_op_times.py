"""The split of a run's device time by op kind (pq_result gate_ms, noise_ms,
phase_ms) and by gate (pq_result_gates): every kind that ran has its share, and
the shares add up to the sweep's time, for runs of one block, of the grid, and
of a batch."""

from __future__ import annotations

import math

import pytest
from harness import from_circuit, from_workload, make_cfg, run_gpu_batch

from propaq_b200 import _native, workloads
from propaq_b200.circuits import PauliCircuit, PauliRotation
from propaq_b200.datatypes import PauliString, PauliTermSum

pytestmark = pytest.mark.gpu


def with_phases():
    """A 5 x 5 kicked Ising circuit with rotations by pi, noise after every layer."""
    wl = workloads.kicked_ising(5, 5, 5)
    pi = [PauliRotation(PauliString(1 << q, 0, 25), math.pi) for q in range(0, 25, 3)]
    p = from_circuit(0, 25, PauliTermSum({PauliString(0, 1 << 12, 25): 1.0}),
                     PauliCircuit([layer + pi for layer in wl.circuit.layers]), 0, max_weight=10, min_coeff=1e-5)
    p.noise_table = from_workload(wl).noise_table
    return p


@pytest.mark.parametrize("make", [lambda: from_workload(workloads.kicked_ising(2, 2, 4)),
                                  lambda: from_workload(workloads.kicked_ising(6, 6, 6)), with_phases],
                         ids=["solo", "grid", "phases"])
def test_shares_add_up(make):
    p = make()
    engine = _native.Engine(0)
    cfg, keep = make_cfg(p, want_terms=False)
    for _ in range(2):  # the second run has nothing to grow
        res, _ = engine.run(cfg, p.obs_keys, p.obs_coeffs, p.gate_keys, p.angles, p.offsets, p.diag)
    for ops, ms in ((res.gate_ops, res.gate_ms), (res.noise_ops, res.noise_ms), (res.phase_ops, res.phase_ms)):
        assert (ms > 0.0) == (ops > 0)
    total = res.gate_ms + res.noise_ms + res.phase_ms
    # the stamps leave out the launches themselves, tens of microseconds
    assert 0.5 * res.sweep_ms - 0.1 < total < 1.05 * res.sweep_ms + 0.01
    gates = engine.gates()
    assert all(g.elapsed_ms > 0.0 for g in gates if g.op >= 0)
    assert abs(sum(g.elapsed_ms for g in gates) - res.gate_ms - res.phase_ms) < 1e-6 + 1e-9 * total


def test_shares_in_a_batch(gpu_engine):
    # solo starts side by side, then one instance after another: no instance is
    # given the time of those before it
    probs = [from_workload(workloads.kicked_ising(6, 6, 6, 0.3 + 0.1 * i)) for i in range(4)]
    probs.append(from_workload(workloads.kicked_ising(2, 2, 4)))
    run_gpu_batch(gpu_engine, probs, want_terms=False)
    results = [g.res for g in run_gpu_batch(gpu_engine, probs, want_terms=False)]
    assert all(r.gate_ms > 0.0 and r.noise_ms > 0.0 for r in results)
    total = sum(r.gate_ms + r.noise_ms + r.phase_ms for r in results)
    assert total < 1.2 * results[0].device_ms + 0.1
