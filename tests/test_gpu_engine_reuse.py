"""A run's results, and the memory it may use, do not depend on what its engine
ran before it."""

from __future__ import annotations

import gc

import numpy as np
import pytest
from harness import assert_terms_equal, from_circuit, from_workload, make_cfg, run_gpu, run_oracle

from propaq_b200 import _native, workloads
from propaq_b200.circuits import PauliCircuit, PauliRotation
from propaq_b200.datatypes import PauliString, PauliTermSum

pytestmark = pytest.mark.gpu


def run(engine, p, **knobs):
    cfg, keep = make_cfg(p, want_terms=False)
    for k, v in knobs.items():
        setattr(cfg, k, v)
    return engine.run(cfg, p.obs_keys, p.obs_coeffs, p.gate_keys, p.angles, p.offsets, p.diag)


def test_key_bytes_leave_out_another_runs_table():
    p = from_workload(workloads.tfim_chain(12, 4))
    fresh = run(_native.Engine(0), p)[0]
    engine = _native.Engine(0)
    # a knob at its default takes the row sweep, whose hash table stays allocated
    row = run(engine, from_workload(workloads.kicked_ising(4, 4, 6)), fuse_max=2)[0]
    after, nt = run(engine, p)
    assert row.sparse_key_bytes > row.n_final * 8
    assert after.sparse_key_bytes == fresh.sparse_key_bytes == fresh.n_final * 8
    assert np.array_equal(nt, run(engine, p)[1])


def test_idle_bins_make_room_for_other_runs(oracle):
    # A binned run leaves its bins (2 x 21 MB) in the engine; a run that may
    # not take half a megabyte more, and needs 3 MB of rows and hash table,
    # gets theirs.
    p = from_workload(workloads.tfim_chain(20, 10))
    engine = _native.Engine(0)
    run(engine, p)
    held = engine.device_bytes()
    engine.set_limits(max_device_bytes=held + (1 << 19))
    g = run_gpu(engine, p)  # a byte limit takes the row sweep
    assert engine.device_bytes() < held - (30 << 20)
    o = run_oracle(oracle, p)
    assert np.array_equal(g.n_terms, o.n_terms)
    assert_terms_equal(g.keys, g.coeffs, o.keys, o.coeffs)
    engine.set_limits()
    g = run_gpu(engine, p)
    assert np.array_equal(g.n_terms, o.n_terms)
    assert_terms_equal(g.keys, g.coeffs, o.keys, o.coeffs)


def test_terms_without_room_to_sort_them():
    # 2^21 terms of 4 words.  With next to no device memory left, the scratch
    # their sort takes (150 MB and more) is not there even with the idle bins
    # given back, and the host sorts them: the same terms in the same order.
    import torch

    n, width = 21, 120
    rng = np.random.default_rng(3)
    x = [PauliRotation(PauliString(1 << q, 0, width), float(a)) for q, a in enumerate(rng.uniform(0.3, 1.2, n))]
    p = from_circuit(0, width, PauliTermSum({PauliString(0, (1 << n) - 1, width): 1.0}), PauliCircuit([x]), 0)
    want = run_gpu(_native.Engine(0), p)
    engine = _native.Engine(0)
    run(engine, p)
    gc.collect()
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - (4 << 20), dtype=torch.uint8, device="cuda")
    try:
        g = run_gpu(engine, p)
    finally:
        del held
        torch.cuda.empty_cache()
    assert g.n_final == 1 << n
    assert np.array_equal(g.keys, want.keys) and np.array_equal(g.coeffs, want.coeffs)
