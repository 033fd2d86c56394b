"""4-cycles counted by several slabs of bit rows.  The inputs are chosen so that
the slabs pay (recomputed here from the rule in c4_rows.cuh and asserted): a
core of some slabs, a block in which counters reach every width, and vertices w
below, inside and above the slabs.  Against the CPU oracle."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SLAB, WEDGES, MOST = 4096, 10, 8  # kC4RowIds, kC4RowWedges, kC4MaxSlabs
WIDTHS = [2, 7, 8, 9, 30, 31, 32, 33, 223, 224, 225, 254, 255, 256, 257, 700]


def slabs_that_pay(ptr, idx, n):
    """Slabs from the top whose tops have at least WEDGES wedges per row read."""
    deg = np.diff(ptr.astype(np.int64))
    rank = np.empty(n, np.int64)
    rank[np.lexsort((np.arange(n), deg))] = np.arange(n)
    v, u = rank[np.repeat(np.arange(n), deg)], rank[idx.astype(np.int64)]
    order = np.lexsort((u, v))
    v, u = v[order], u[order]
    first = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(v, minlength=n), out=first[1:])
    pos = np.arange(v.size) - first[v]  # neighbours of v below u
    up = u > v
    wedges = np.bincount((n - 1 - u[up]) // SLAB, weights=pos[up], minlength=MOST)[:MOST]
    rows = int(deg[deg >= 2].sum())
    k = 0
    while k < min(MOST, -(-n // SLAB)) and wedges[k] and wedges[k] // WEDGES >= rows:
        k += 1
    return k


def core_with_widths(n, degree, seed, tail=0):
    """A random core of n vertices, a complete block in it, and for every width d
    three vertices adjacent to the first d of the block's one side: they share d
    neighbours with each vertex of the other side.  `tail` vertices beside it."""
    rng = np.random.default_rng(seed)
    src, dst = [rng.integers(0, n, n * degree // 2)], [rng.integers(0, n, n * degree // 2)]
    side = rng.permutation(n)
    a, b = side[:40], side[40:40 + max(WIDTHS)]
    src.append(np.repeat(a, b.size))
    dst.append(np.tile(b, a.size))
    at = n
    for d in WIDTHS:
        for _ in range(3):
            src.append(np.full(d, at))
            dst.append(b[:d])
            at += 1
    if tail:  # a sparse part: edges among themselves, and a few into the core
        src += [rng.integers(at, at + tail, 2 * tail), rng.integers(at, at + tail, tail // 2)]
        dst += [rng.integers(at, at + tail, 2 * tail), rng.integers(0, n, tail // 2)]
        at += tail
    return np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32), at


@pytest.mark.parametrize("n,degree,tail,slabs", [
    (3000, 60, 0, 1),          # less than a slab
    (SLAB - 48, 90, 0, 1),     # exactly one, with the 48 others
    (SLAB + 1, 100, 500, 1),
    (2 * SLAB, 200, 0, 1),
    (2 * SLAB, 700, 0, 2),
    (3 * SLAB - 47, 240, 3000, 2),
    (20011, 300, 0, 3),
    (20011, 420, 9000, 3),
])
def test_slabs_that_pay(cuda, n, degree, tail, slabs):
    import torch

    src, dst, n = core_with_widths(n, degree, n + degree, tail)
    ptr, idx = O.sym_csr(src, dst, n)
    assert slabs_that_pay(ptr, idx, n) == slabs
    want = O.c4_count(ptr, idx)
    with gb.Graph.upload(ptr, idx, n) as g:
        assert g.count(gb.GARY_PATTERN_4CYCLE) == want
        out = torch.zeros(1, dtype=torch.int64, device="cuda")
        total = 0
        for k in range(3):
            gb._lib.check(gb.load().gary_count_shard_async(g.handle, 4, 0, k, 3, None, out.data_ptr()), "shard")
            total += int(out.item())
        assert total == want
