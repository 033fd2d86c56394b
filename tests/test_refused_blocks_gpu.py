"""A count that is refused a block of device memory ends with GARY_ERR_OOM or
with the right count, whichever block it is, and leaves nothing half built: the
next count of the same graph is right.  Every block of every plan is refused in
turn ("refuse_block"), against the CPU oracle."""
from __future__ import annotations

import ctypes as C

import pytest

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

BLOCKS = 48  # more than any plan asks for


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


def _refuse(k):
    gb._lib.check(gb.load().gary_tune(b"refuse_block", k), "refuse_block")


@pytest.mark.parametrize("pattern", [gb.GARY_PATTERN_TRIANGLE, gb.GARY_PATTERN_4CYCLE, gb.GARY_PATTERN_4CLIQUE])
def test_counts_with_a_block_refused(cuda, skewed, pattern):
    ptr, idx, n, want = skewed
    lib = gb.load()
    refused = 0
    for k in range(1, BLOCKS):
        with gb.Graph.upload(ptr, idx, n) as g:
            out = C.c_uint64(0)
            _refuse(k)
            try:
                rc = lib.gary_count(g.handle, pattern, 0, None, C.byref(out))
            finally:
                _refuse(0)
            assert rc in (gb._lib.GARY_OK, gb._lib.GARY_ERR_OOM), (k, lib.gary_last_error())
            if rc == gb._lib.GARY_OK:
                assert out.value == want[pattern], k
            else:
                refused += 1
            assert g.count(pattern) == want[pattern], k
    # a plan that is refused a block is made again without rows: only blocks that
    # no plan can do without end a count, never all of them
    assert refused < BLOCKS // 2


@pytest.mark.parametrize("k", [1, 2])
def test_coo_view_with_a_block_refused(cuda, skewed, k):
    """The COO view is refused its row or its column array: the next call builds both."""
    ptr, idx, n, _ = skewed
    with gb.Graph.upload(ptr, idx, n) as g:
        _refuse(k)
        try:
            with pytest.raises(gb.GaryError):
                g.device_coo()
        finally:
            _refuse(0)
        coo = g.device_coo()
        assert coo.rowIdx and coo.colIdx
        p, i, _ = g.download()
        assert int(p[-1]) == len(i) == len(idx) // 2
