"""4-clique counts through adjacency rows over the top 16384 ids: graphs just
below, at and above that size, vertices with few top neighbours (rows missing,
up to and past the eighth at which a vertex stops using rows), every class of
worker.  Against the CPU oracle and closed forms."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOP = 16384  # kAdjRowIds in hub.cuh


def _graph(n, k_lo, k_hi, low, top_edges, seed):
    """A dense top of TOP vertices, and n - TOP others with k_lo..k_hi skewed
    edges into it and `low` among themselves."""
    rng = np.random.default_rng(seed)
    t = min(TOP, n)
    m = n - t
    src, dst = [rng.integers(0, t, top_edges)], [(t * rng.random(top_edges) ** 3).astype(np.int64)]
    if m:
        k = rng.integers(k_lo, k_hi + 1, m)
        src += [np.repeat(np.arange(t, n), k), np.repeat(np.arange(t, n), low)]
        dst += [(t * rng.random(int(k.sum())) ** 3).astype(np.int64), rng.integers(t, n, m * low)]
    return np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32)


@pytest.mark.parametrize("n,k_lo,k_hi,low,top_edges", [
    (TOP - 1, 0, 0, 0, 500000),
    (TOP, 0, 0, 0, 500000),
    (TOP + 1, 20, 20, 0, 500000),
    (TOP + 3000, 12, 22, 6, 400000),     # rows of some, none of others
    (TOP + 9000, 2, 60, 25, 500000),     # long low parts: hash and rows meet inside a word
    (TOP + 2500, 130, 420, 40, 900000),  # CTA classes
])
def test_four_cliques_through_rows(cuda, n, k_lo, k_hi, low, top_edges):
    src, dst = _graph(n, k_lo, k_hi, low, top_edges, n)
    ptr, idx = O.sym_csr(src, dst, n)
    optr, oidx = O.orient(ptr, idx)
    with gb.Graph.upload(ptr, idx, n) as g:
        assert g.count(gb.GARY_PATTERN_4CLIQUE) == O.k4_count(optr, oidx)


@pytest.mark.parametrize("k", [3, 4, 31, 32, 33, 64, 129, 363, 900])
@pytest.mark.parametrize("extra", [0, 40000])
def test_complete_graphs_beside_isolated_vertices(cuda, k, extra):
    """K_k with `extra` vertices of degree 0 below it (so that n passes TOP)."""
    n = k + extra
    i, j = np.triu_indices(k, 1)
    ptr, idx = O.sym_csr((i + extra).astype(np.uint32), (j + extra).astype(np.uint32), n)
    with gb.Graph.upload(ptr, idx, n) as g:
        assert g.count(gb.GARY_PATTERN_4CLIQUE) == k * (k - 1) * (k - 2) * (k - 3) // 24
