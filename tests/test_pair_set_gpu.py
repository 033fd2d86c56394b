"""Middle vertices whose higher neighbours lie too far apart for a bitmap
(spans beyond 32 K ids): pair sets of every table size up to the largest, with
evictions (the fullest tables hold 512 ids in 2048 slots), and ids at both ends
of what 16-bit entries hold.  Against the CPU oracle."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,per_vertex", [(40000, 12), (40000, 40), (36001, 150), (36001, 290)])
def test_wide_lists_of_every_length(cuda, n, per_vertex):
    """Out-degrees run from 0 to about twice per_vertex in the degree order."""
    src, dst = gb.gen_er(n, n * per_vertex, per_vertex)
    ptr, idx = gb.csr_from_edges(src, dst, n)
    optr, oidx = O.orient(ptr, idx)
    with gb.Graph.upload(ptr, idx, n) as g:
        assert g.count() == O.tri_count(optr, oidx)


@pytest.mark.parametrize("n", [(0xFFFF << 6) - 1, 0xFFFF << 6, (0xFFFF << 6) + 70, 1 << 22, (1 << 22) + 3])
def test_ids_at_the_entry_limit(cuda, n):
    """Entries are id >> k, and 0xFFFF is an empty slot: the smallest table
    (k = 6) must not be used once an id below n has that entry.  A sparse graph
    of n vertices whose last ranks form the wide lists."""
    rng = np.random.default_rng(n)
    core = 70000
    m = core * 20
    src = rng.integers(n - core, n, m).astype(np.uint32)
    dst = rng.integers(n - core, n, m).astype(np.uint32)
    ptr, idx = gb.csr_from_edges(src, dst, n)
    optr, oidx = O.orient(ptr, idx)
    with gb.Graph.upload(ptr, idx, n) as g:
        assert g.count() == O.tri_count(optr, oidx)
