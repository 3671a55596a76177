"""A run's results, and the memory it may use, do not depend on what its engine
ran before it."""

from __future__ import annotations

import numpy as np
import pytest
from harness import assert_terms_equal, from_workload, make_cfg, run_gpu, run_oracle

from propaq_b200 import _native, workloads

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
