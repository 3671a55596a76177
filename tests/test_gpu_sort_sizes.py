"""Sorted term output (propaq_b200/csrc/pq_sort.cu) at the edges of its paths:
one counting launch up to 2^14 rows, radix passes over tiles of 256 rows up to
2^17 and of 2,048 beyond.  A run without gates returns its observable's terms in
key order, whatever order they came in."""

from __future__ import annotations

import numpy as np
import pytest
from harness import Problem, run_gpu

pytestmark = pytest.mark.gpu


def observable(n_terms, W, seed):
    """n_terms distinct keys that differ in few words and few digits, shuffled."""
    rng = np.random.default_rng(seed)
    keys = np.zeros((n_terms, W), dtype=np.uint64)
    ids = rng.permutation(n_terms).astype(np.uint64)
    keys[:, 0] = ids * np.uint64(0x101) % np.uint64(1 << 20)
    keys[:, W - 1] ^= ids << np.uint64(40)
    return keys, rng.normal(size=n_terms)


@pytest.mark.parametrize("W", [1, 2, 4, 8])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 4097, 16383, 16384, 16385, 40000, 131072, 131073])
@pytest.mark.parametrize("sort", [False, True], ids=["plain", "sorted"])
def test_terms_in_key_order(gpu_engine, W, n, sort):
    keys, coeffs = observable(n, W, 10 * n + W)
    p = Problem(0, 32 * W, W, keys, coeffs, np.zeros((0, W), np.uint64), np.zeros(0), np.zeros(1, np.uint32), None)
    g = run_gpu(gpu_engine, p, sort_terms=sort)
    order = np.lexsort(keys.T)  # last word most significant
    assert np.array_equal(g.keys, keys[order])
    assert np.array_equal(g.coeffs, coeffs[order])
