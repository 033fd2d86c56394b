"""Plans with bit rows and plans made without them, for want of memory, count
the same: against the CPU oracle, for all three patterns, with the rows' memory
seen to be there or not."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MB = 1 << 20


class _Held:
    """Device bytes a plan holds, with nothing cached beside it."""

    def __enter__(self):
        torch.cuda.empty_cache()
        gb.load().gary_tune(b"pool_keep_bytes", 0)  # freed blocks go back to the driver
        return self

    def __exit__(self, *_):
        gb.load().gary_tune(b"refuse_block", 0)
        gb.load().gary_tune(b"pool_keep_bytes", (1 << 64) - 1)

    def plan_bytes(self, g, pattern, want, refuse=0):
        """Of a plan built for a count of `pattern`, which has to be right."""
        gb._lib.check(gb.load().gary_graph_drop_plans(g.handle), "drop plans")
        free = self.free()
        gb._lib.check(gb.load().gary_tune(b"refuse_block", refuse), "refuse_block")
        assert g.count(pattern) == want
        gb._lib.check(gb.load().gary_tune(b"refuse_block", 0), "refuse_block")
        return free - self.free()

    def free(self):
        torch.cuda.synchronize()
        gb.load().gary_tune(b"pool_keep_bytes", 0)  # scratch that was freed goes back as well
        return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("pattern", [gb.GARY_PATTERN_TRIANGLE, gb.GARY_PATTERN_4CYCLE, gb.GARY_PATTERN_4CLIQUE])
def test_a_plan_refused_its_rows_counts_without(cuda, pattern):
    scale = 16
    src, dst = gb.gen_rmat(scale, 21, 24 << scale)
    ptr, idx = O.sym_csr(src, dst, 1 << scale)
    optr, oidx = O.orient(ptr, idx)
    want = {3: lambda: O.tri_count(optr, oidx), 4: lambda: O.c4_count(ptr, idx),
            5: lambda: O.k4_count(optr, oidx)}[pattern]()
    with _Held() as held, gb.Graph.upload(ptr, idx, 1 << scale) as g:
        assert g.count(pattern) == want  # the symmetric lists and the result word are there from now on
        bytes_, tiles = [], []
        for refuse in (0, 1, 0):  # the first block of a plan is one of its rows'
            bytes_.append(held.plan_bytes(g, pattern, want, refuse))
            tiles.append(g.last_stats()["tiles"])
        if pattern == gb.GARY_PATTERN_4CLIQUE:  # a row of 16384 bits for each of 16384 vertices at least
            assert min(bytes_[0], bytes_[2]) - bytes_[1] >= 2048 * 16384, bytes_
        else:  # what rows count is in no tile
            assert tiles[0] < tiles[1] and tiles[0] == tiles[2], tiles


def test_four_cliques_without_room_for_rows(cuda):
    """Rows of 150 MB, refused by the driver, and rows of more than 1 GB, which ask
    for twice their room."""
    top = 16384
    for low, room, rows in ((60000, 100 * MB, 150 * MB), (560000, 1500 * MB, 1100 * MB)):
        rng = np.random.default_rng(low)
        src = np.concatenate([rng.integers(0, top, 600000), np.repeat(np.arange(top, top + low), 20)])
        dst = np.concatenate([(top * rng.random(600000) ** 4).astype(np.int64), rng.integers(0, top, low * 20)])
        _check_without_room(src, dst, top + low, gb.GARY_PATTERN_4CLIQUE, None, room, rows)


def test_four_cycles_without_room_for_rows(cuda):
    """Groups of vertices that share the same 48 tops, a slab of 200 MB: a group of
    g has C(g, 2) C(48, 2) cycles."""
    sets, low = 4096 // 48, 400000
    v = np.repeat(np.arange(4096, 4096 + low), 48)
    src, dst = v, v % sets * 48 + np.tile(np.arange(48), low)
    g = np.bincount(np.arange(4096, 4096 + low) % sets)
    _check_without_room(src, dst, 4096 + low, gb.GARY_PATTERN_4CYCLE, int((g * (g - 1) // 2).sum()) * (48 * 47 // 2),
                        150 * MB, 200 * MB)


def _check_without_room(src, dst, n, pattern, want, room, rows):
    ptr, idx = gb.csr_from_edges(src.astype(np.uint32), dst.astype(np.uint32), n)
    want = O.k4_count(*O.orient(ptr, idx)) if want is None else want
    with _Held() as held, gb.Graph.upload(ptr, idx, n) as g:
        assert g.count(pattern) == want
        assert held.plan_bytes(g, pattern, want) >= rows
        gb._lib.check(gb.load().gary_graph_drop_plans(g.handle), "drop plans")
        full = torch.empty(held.free() - room, dtype=torch.uint8, device="cuda")
        try:
            assert held.plan_bytes(g, pattern, want) < rows // 2
        finally:
            del full
            torch.cuda.empty_cache()
