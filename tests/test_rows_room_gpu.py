"""Bit rows are an option of a plan: on a device with no room for them the same
counts come from plans without rows."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ROOM = 400 << 20  # less than twice the rows below: 4-cliques 1 GB, 4-cycles 250 MB a slab


def test_counts_without_room_for_rows(cuda):
    top, low = 16384, 500000
    rng = np.random.default_rng(5)
    k = rng.integers(16, 24, low)
    src = np.concatenate([rng.integers(0, top, 400000), np.repeat(np.arange(top, top + low), k)])
    dst = np.concatenate([rng.integers(0, top, 400000), rng.integers(0, top, int(k.sum()))])
    ptr, idx = O.sym_csr(src.astype(np.uint32), dst.astype(np.uint32), top + low)
    patterns = (gb.GARY_PATTERN_4CLIQUE, gb.GARY_PATTERN_4CYCLE)
    with gb.Graph.upload(ptr, idx, top + low) as g:
        want = [g.count(p) for p in patterns]
        lib = gb._lib.load()
        gb._lib.check(lib.gary_graph_drop_plans(g.handle), "drop plans")
        torch.cuda.empty_cache()
        lib.gary_tune(b"pool_keep_bytes", 0)  # blocks of the dropped plans go back to the driver
        full = torch.empty(torch.cuda.mem_get_info()[0] - ROOM, dtype=torch.uint8, device="cuda")
        try:
            assert [g.count(p) for p in patterns] == want
        finally:
            del full
            torch.cuda.empty_cache()
            lib.gary_tune(b"pool_keep_bytes", (1 << 64) - 1)
