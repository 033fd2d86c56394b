"""Shards are counted by processes that each build a plan of their own, so what
a shard covers must be the same in every build of the plan: shard k of N from
one upload and the other shards from others add up to the oracle's count."""
from __future__ import annotations

import pytest

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _shard(g, pattern, shard, nshards):
    import torch

    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    gb._lib.check(gb.load().gary_count_shard_async(g.handle, pattern, 0, shard, nshards, None, out.data_ptr()), "shard")
    return int(out.item())


@pytest.mark.parametrize("scale,ef", [(12, 16), (15, 11), (17, 16)])
@pytest.mark.parametrize("tune", [{}, {"warp_cap": 8, "cta_tile_cost": 2048}])  # split vertices; CTA tiles as well
def test_shards_of_separate_triangle_plans_add_up(cuda, scale, ef, tune):
    src, dst = gb.gen_rmat(scale, scale + ef, ef << scale)
    ptr, idx = O.sym_csr(src, dst, 1 << scale)
    optr, oidx = O.orient(ptr, idx)
    want = O.tri_count(optr, oidx)
    lib = gb.load()
    try:
        for key, value in tune.items():
            gb._lib.check(lib.gary_tune(key.encode(), value), key)
        for nshards in (2, 3, 5, 8):
            for _ in range(3):
                total = 0
                for k in range(nshards):
                    with gb.Graph.upload(ptr, idx, 1 << scale) as g:
                        total += _shard(g, gb.GARY_PATTERN_TRIANGLE, k, nshards)
                assert total == want, (nshards, total - want)
    finally:
        lib.gary_tune(b"reset", 0)


def test_shards_of_plans_with_many_record_tiles(cuda):
    """Lists of more than 2^14 tiles of 2048 padded words (one octet a vertex at
    least), a skewed core among them."""
    import numpy as np

    n = 5_000_000
    rng = np.random.default_rng(14)
    s, d = gb.gen_rmat(16, 3, 1 << 20)
    src = np.concatenate([s, rng.integers(0, n, 3 * n, dtype=np.uint32)])
    dst = np.concatenate([d, rng.integers(0, n, 3 * n, dtype=np.uint32)])
    ptr, idx = gb.csr_from_edges(src, dst, n)
    optr, oidx = O.orient(ptr, idx)
    assert int(((np.diff(optr.astype(np.int64)) + 7) // 8).sum()) * 8 > 2048 << 14
    want = O.tri_count(optr, oidx)
    total = 0
    for k in range(3):
        with gb.Graph.upload(ptr, idx, n) as g:
            total += _shard(g, gb.GARY_PATTERN_TRIANGLE, k, 3)
    assert total == want
