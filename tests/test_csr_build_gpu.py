"""gary_csr_from_edges on lists of every awkward shape, against the oracle's
symmetric CSR: nothing kept, one edge many times, loops between copies of an
edge, tiles of the compaction cut anywhere, isolated vertices at both ends."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TILE = 4096  # keys a CTA compacts at a time


@pytest.mark.parametrize("m", [0, 1, 2, 255, TILE - 1, TILE, TILE + 1, 3 * TILE + 17, 200003])
@pytest.mark.parametrize("kind", ["sparse", "dense", "loops", "one", "hub"])
def test_matches_the_oracle(cuda, m, kind):
    rng = np.random.default_rng(m + len(kind))
    n = {"sparse": 100003, "dense": 70, "loops": 50, "one": 9, "hub": 65536}[kind]
    s, d = rng.integers(0, n, m), rng.integers(0, n, m)
    if kind == "loops":
        d = np.where(rng.random(m) < 0.8, s, d)
    elif kind == "one":
        s, d = np.full(m, 7), np.where(rng.random(m) < 0.5, 7, 3)
    elif kind == "hub":
        s = np.where(rng.random(m) < 0.5, n - 1, s)
    s, d = s.astype(np.uint32), d.astype(np.uint32)
    want_ptr, want_idx = O.sym_csr(s, d, n)
    ptr, idx = gb.csr_from_edges(s, d, n)
    assert np.array_equal(ptr, want_ptr) and np.array_equal(idx, want_idx)


@pytest.mark.parametrize("n", [1, 2, (1 << 16) + 1, (1 << 24) + 5])
def test_vertex_counts_around_the_key_widths(cuda, n):
    rng = np.random.default_rng(n)
    m = 5000
    s, d = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    s[:2], d[:2] = [0, n - 1], [n - 1, 0]
    want_ptr, want_idx = O.sym_csr(s, d, n)
    ptr, idx = gb.csr_from_edges(s, d, n)
    assert np.array_equal(ptr, want_ptr) and np.array_equal(idx, want_idx)
    bad = d.copy()
    bad[4321] = n
    with pytest.raises(gb.GaryError):
        gb.csr_from_edges(s, bad, n)
