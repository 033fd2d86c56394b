"""Triangle counts on graphs whose hub rows are used (the top 4096 ranks as bit
rows), at the sizes where they can go wrong, against the CPU oracle: the
smallest graph that has them, lists with a hub neighbour more or less than a
row needs, cuts at every offset within an octet, middle vertices without a
row, hubs counted as the lowest vertex, and every shard split."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

HUBS = 4096      # kHubIds in hub.cuh
ROW_MIN = 64     # kHubMin


def _core_periphery(n, k_lo, k_hi, low, hub_edges, seed):
    """Hubs are caller ids 0..HUBS-1; every other vertex takes k_lo..k_hi of
    them and `low` of its peers; the hubs share hub_edges random edges."""
    rng = np.random.default_rng(seed)
    m = n - HUBS
    k = rng.integers(k_lo, k_hi + 1, m)
    src = np.repeat(np.arange(HUBS, n), k)
    # cubed, so that a few hubs are everywhere and rows are unevenly dense
    dst = (HUBS * rng.random(src.size) ** 3).astype(np.int64)
    src = np.concatenate([src, np.repeat(np.arange(HUBS, n), low), rng.integers(0, HUBS, hub_edges)])
    dst = np.concatenate([dst, rng.integers(HUBS, n, m * low), rng.integers(0, HUBS, hub_edges)])
    return src.astype(np.uint32), dst.astype(np.uint32)


@pytest.mark.parametrize("n,k_lo,k_hi,low,hub_edges", [
    (2 * HUBS, 70, 90, 3, 400000),          # one vertex too few for hub rows
    (2 * HUBS + 1, 70, 90, 3, 400000),      # the smallest graph with them
    (12001, ROW_MIN - 2, ROW_MIN + 6, 9, 100000),   # on both sides of the row limit
    (12289, 40, 200, 20, 0),                # cuts at every octet offset, hubs without edges of their own
    (9001, 90, 160, 0, 600000),             # empty low parts
    (30011, 4, 70, 12, 900000),             # mostly middle vertices without a row; hubs counted as u
])
def test_hub_rows_match_the_oracle(cuda, n, k_lo, k_hi, low, hub_edges):
    import torch

    src, dst = _core_periphery(n, k_lo, k_hi, low, hub_edges, n)
    ptr, idx = O.sym_csr(src, dst, n)
    optr, oidx = O.orient(ptr, idx)
    want = O.tri_count(optr, oidx)
    with gb.Graph.upload(ptr, idx, n) as g:
        assert g.count() == want
        out = torch.zeros(1, dtype=torch.int64, device="cuda")
        total = 0
        for k in range(3):
            gb._lib.check(gb.load().gary_count_shard_async(g.handle, 3, 0, k, 3, None, out.data_ptr()), "shard")
            total += int(out.item())
        assert total == want
