"""4-cycles under the top ids counted by bit rows (slabs of 4096 ids): graphs of
less than a slab, one slab and a few, vertices w inside, below and between
slabs, degrees around the counters' widths, and every shard split.  Against the
CPU oracle and closed forms."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SLAB = 4096


def _skewed(n, m, power, seed):
    """Edges whose one end is drawn towards low caller ids."""
    rng = np.random.default_rng(seed)
    return (n * rng.random(m) ** power).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)


def _check(ptr, idx, n):
    import torch

    want = O.c4_count(ptr, idx)
    with gb.Graph.upload(ptr, idx, n) as g:
        assert g.count(gb.GARY_PATTERN_4CYCLE) == want
        out = torch.zeros(1, dtype=torch.int64, device="cuda")
        total = 0
        for k in range(3):
            gb._lib.check(gb.load().gary_count_shard_async(g.handle, 4, 0, k, 3, None, out.data_ptr()), "shard")
            total += int(out.item())
        assert total == want


@pytest.mark.parametrize("n", [50, SLAB - 1, SLAB, SLAB + 1, 2 * SLAB + 1, 3 * SLAB, 30011])
@pytest.mark.parametrize("power", [1, 4])
def test_graphs_around_the_slabs(cuda, n, power):
    src, dst = _skewed(n, 24 * n, power, n + power)
    ptr, idx = O.sym_csr(src, dst, n)
    _check(ptr, idx, n)


@pytest.mark.parametrize("deg", [2, 7, 8, 9, 30, 31, 32, 33, 223, 224, 225, 254, 255, 256, 257, 700])
def test_degrees_at_the_counter_widths(cuda, deg):
    """K_{a,deg}: every left vertex has degree deg, and every pair of left
    vertices deg common neighbours; plus a sparse graph beside it."""
    a, extra = 300, 9000
    n = a + deg + extra
    s, d = np.repeat(np.arange(a), deg), a + np.tile(np.arange(deg), a)
    rng = np.random.default_rng(deg)
    s = np.concatenate([s, rng.integers(a + deg, n, 2 * extra)])
    d = np.concatenate([d, rng.integers(a + deg, n, 2 * extra)])
    ptr, idx = O.sym_csr(s.astype(np.uint32), d.astype(np.uint32), n)
    _check(ptr, idx, n)
