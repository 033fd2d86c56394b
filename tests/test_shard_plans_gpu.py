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


@pytest.mark.parametrize("n,tiles", [(5_000_000, 1 << 14), (17_500_000, 1 << 16)])
def test_shards_of_plans_with_many_record_tiles(cuda, n, tiles):
    """Lists of more than 2^14 and more than 2^16 tiles of 2048 padded words: a
    ring (one octet a vertex) with a skewed core."""
    import numpy as np

    s, d = gb.gen_rmat(16, 3, 1 << 20)
    ring = np.arange(n, dtype=np.uint32)
    src, dst = np.concatenate([s, ring]), np.concatenate([d, np.roll(ring, 1)])
    ptr, idx = gb.csr_from_edges(src, dst, n)
    optr, oidx = O.orient(ptr, idx)
    assert int(((np.diff(optr.astype(np.int64)) + 7) // 8).sum()) * 8 > 2048 * tiles
    want = O.tri_count(optr, oidx)
    total = 0
    for k in range(3):
        with gb.Graph.upload(ptr, idx, n) as g:
            total += _shard(g, gb.GARY_PATTERN_TRIANGLE, k, 3)
    assert total == want


@pytest.fixture(scope="module")
def skewed():
    """A graph whose plans have bit rows, for all three patterns."""
    scale = 15
    src, dst = gb.gen_rmat(scale, 7, 24 << scale)
    ptr, idx = O.sym_csr(src, dst, 1 << scale)
    optr, oidx = O.orient(ptr, idx)
    return ptr, idx, 1 << scale, {gb.GARY_PATTERN_TRIANGLE: O.tri_count(optr, oidx),
                                  gb.GARY_PATTERN_4CYCLE: O.c4_count(ptr, idx),
                                  gb.GARY_PATTERN_4CLIQUE: O.k4_count(optr, oidx)}


PATTERNS = [gb.GARY_PATTERN_TRIANGLE, gb.GARY_PATTERN_4CYCLE, gb.GARY_PATTERN_4CLIQUE]
BLOCKS = 40  # more than any plan asks for


def _refuse(k):
    gb._lib.check(gb.load().gary_tune(b"refuse_block", k), "refuse_block")


def _shard_or_oom(g, pattern, shard, nshards):
    import torch

    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    rc = gb.load().gary_count_shard_async(g.handle, pattern, 0, shard, nshards, None, out.data_ptr())
    if rc == gb._lib.GARY_ERR_OOM:
        return None
    gb._lib.check(rc, "shard")
    return int(out.item())


@pytest.mark.parametrize("pattern", PATTERNS)
@pytest.mark.parametrize("whole_first", [False, True])
def test_a_shard_does_not_depend_on_free_memory(cuda, skewed, pattern, whole_first):
    """A rank that is refused a block of its plan, be it one of the bit rows
    which a count can do without, counts the shard the other rank leaves to it,
    or ends with GARY_ERR_OOM: never another part of the graph."""
    ptr, idx, n, want = skewed
    with gb.Graph.upload(ptr, idx, n) as g:
        other = _shard(g, pattern, 1, 2)
    for k in range(1, BLOCKS):
        with gb.Graph.upload(ptr, idx, n) as g:
            _refuse(k)
            try:
                if whole_first:  # leaves a plan without rows behind
                    try:
                        assert g.count(pattern) == want[pattern]
                    except gb.GaryError:
                        pass
                mine = _shard_or_oom(g, pattern, 0, 2)
            finally:
                _refuse(0)
            if mine is not None:
                assert mine + other == want[pattern], k
            assert _shard(g, pattern, 0, 2) + other == want[pattern], k
            assert g.count(pattern) == want[pattern], k


@pytest.mark.parametrize("pattern", PATTERNS)
@pytest.mark.parametrize("nshards", [2, 3, 7])
def test_shards_of_separate_plans_add_up(cuda, skewed, pattern, nshards):
    ptr, idx, n, want = skewed
    total = 0
    for k in range(nshards):
        with gb.Graph.upload(ptr, idx, n) as g:
            if k & 1:  # a plan for whole counts is there already
                assert g.count(pattern) == want[pattern]
            total += _shard(g, pattern, k, nshards)
    assert total == want[pattern]


def test_four_cycle_shards_with_fewer_slabs_than_whole_counts(cuda):
    """Slabs of some 80 MB each: a shard takes those within 128 MB, a whole count
    all that pay, before, between and after the shards."""
    scale = 18
    src, dst = gb.gen_rmat(scale, 18, 16 << scale)
    ptr, idx = O.sym_csr(src, dst, 1 << scale)
    want = O.c4_count(ptr, idx)
    total = 0
    for k in range(3):
        with gb.Graph.upload(ptr, idx, 1 << scale) as g:
            if k == 1:
                assert g.count(gb.GARY_PATTERN_4CYCLE) == want
            total += _shard(g, gb.GARY_PATTERN_4CYCLE, k, 3)
            assert g.count(gb.GARY_PATTERN_4CYCLE) == want
            assert sum(_shard(g, gb.GARY_PATTERN_4CYCLE, j, 2) for j in range(2)) == want
    assert total == want
