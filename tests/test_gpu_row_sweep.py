"""The row sweep's own paths -- class ops, fused pairs, the grid that follows
the live count -- for runs that the binned sweep would take by default.  A
kernel knob at its default value (fuse_max 2) sends a run there with everything
else at its default, so class_ops counts ops that class_op ran and
sweep_launches the sweep's capacity stops and grid changes.  Against the
oracle: live count after every rotation, term set, every coefficient bit for
bit, terms below the cutoff, expectation value."""

from __future__ import annotations

import math

import numpy as np
import pytest
from harness import assert_terms_equal, expectation_close, from_circuit, from_workload, make_cfg, run_oracle
from test_gpu_class import pair_layers, random_obs

from propaq_b200 import _native, workloads
from propaq_b200.circuits import PauliCircuit

pytestmark = pytest.mark.gpu


def row_run(engine, p, want_terms=True, **knobs):
    cfg, keep = make_cfg(p, want_terms)
    for k, v in dict(fuse_max=2, **knobs).items():
        setattr(cfg, k, v)
    res, nt = engine.run(cfg, p.obs_keys, p.obs_coeffs, p.gate_keys, p.angles, p.offsets, p.diag)
    return (res, nt, *(engine.terms(p.n_words) if want_terms else (None, None)))


def check(engine, oracle, p, **knobs):
    res, nt, keys, coeffs = row_run(engine, p, **knobs)
    o = run_oracle(oracle, p)
    assert np.array_equal(nt, o.n_terms), "live counts per gate differ"
    assert int(res.terms_below_cutoff) == o.terms_below_cutoff
    assert_terms_equal(keys, coeffs, o.keys, o.coeffs)
    assert expectation_close(res.expectation_value, o)[0]
    return res


@pytest.mark.parametrize("seed", range(6))
def test_class_ops_on_random_disjoint_layers(gpu_engine, oracle, seed):
    n = [12, 40, 64][seed % 3]
    p = from_circuit(0, n, random_obs(seed, n), PauliCircuit(pair_layers(seed, n, 7)),
                     int(np.random.default_rng(seed).integers(0, 1 << min(n, 60))), max_weight=[4, 6, 10][seed % 3],
                     min_coeff=[1e-3, 1e-5][seed % 2])
    if seed % 2:
        p.noise_table = np.array([math.exp(-0.02 * w) for w in range(n + 1)])
    assert check(gpu_engine, oracle, p).class_ops > 0


def test_class_ops_of_a_workload_and_none_for_generic_angles(gpu_engine, oracle):
    assert check(gpu_engine, oracle, from_workload(workloads.kicked_ising(6, 6, 8))).class_ops > 0
    assert check(gpu_engine, oracle, from_workload(workloads.tfim_chain(20, 10))).class_ops == 0
    assert check(gpu_engine, oracle, from_workload(workloads.kicked_ising(5, 5, 6, max_weight=12))).class_ops == 0


def test_capacity_stops_inside_class_ops_and_fused_pairs(oracle):
    # fresh engines start at 2^16 rows
    res = check(_native.Engine(0), oracle, from_workload(workloads.kicked_ising(10, 10, 6)))
    assert res.class_ops > 0 and res.sweep_launches > 1
    res = check(_native.Engine(0), oracle, from_workload(workloads.kicked_ising(4, 4, 6)))
    assert res.sweep_launches > 3


@pytest.mark.parametrize("make", [lambda: workloads.kicked_ising(6, 6, 6),
                                  lambda: workloads.majorana_givens(n_sites=12, reps=2, seed=4)],
                         ids=["kicked6x6", "majorana12"])
def test_default_grid_grows_with_the_live_count(gpu_engine, oracle, make):
    p = from_workload(make())
    row_run(gpu_engine, p)  # the buffers grow to size here
    auto = check(gpu_engine, oracle, p)
    fixed = check(gpu_engine, oracle, p, blocks_per_sm=3)
    assert auto.peak_terms > 148 * 256
    assert fixed.sweep_launches == 1 < auto.sweep_launches


def test_six_block_build_past_2_24_rows(gpu_engine):
    p = from_workload(workloads.majorana_givens(24, 4))
    row_run(gpu_engine, p, want_terms=False)
    auto, nt = row_run(gpu_engine, p, want_terms=False)[:2]
    fixed, nt_fixed = row_run(gpu_engine, p, want_terms=False, blocks_per_sm=4)[:2]
    assert auto.peak_terms > 1 << 24
    assert fixed.sweep_launches == 1 and auto.sweep_launches >= 4  # 148 x 256, 2^20 and 2^24 rows passed
    assert np.array_equal(nt, nt_fixed)
    assert abs(auto.expectation_value - fixed.expectation_value) <= 1e-13 * max(1.0, abs(fixed.expectation_value))
