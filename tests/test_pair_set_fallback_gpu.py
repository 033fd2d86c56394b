"""Wide lists of middle vertices for which no pair set can be built: ids that
share their place in both tables, and ids of more than 26 bits.  They are
counted with buckets.  Against the CPU oracle and a closed form."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

STEP = 4096   # ids x and x + 2^(2 k) share both places in tables of 2^k slots; k = 6 for lists of up to 32 ids
LEN = 20      # more than two octets, which need no set
RING = 15     # ring neighbours of a top vertex to either side


def _colliding():
    """Vertices u_i, v_i (i < STEP) and STEP * LEN top vertices t.  v_i and u_i
    are adjacent to each other and to t = i, i + STEP, ..; the tops form a ring of
    chords, so that all have one degree and ranks follow ids: u, v, t."""
    top = STEP * LEN
    i, t = np.arange(STEP), np.arange(top)
    src, dst = [i], [STEP + i]
    for first in (0, STEP):
        src.append(np.tile(first + i, LEN))
        dst.append(2 * STEP + t)
    for r in range(1, RING + 1):
        src.append(2 * STEP + t)
        dst.append(2 * STEP + (t + r) % top)
    return np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32), 2 * STEP + top


def _triangles():
    top = STEP * LEN
    # u_i v_i t, LEN each; in the ring, for every t the pairs of chords r + s <= RING
    return STEP * LEN + top * (RING * (RING - 1) // 2)


def test_ids_that_collide_in_both_tables(cuda):
    src, dst, n = _colliding()
    ptr, idx = O.sym_csr(src, dst, n)
    optr, oidx = O.orient(ptr, idx)
    lists = np.split(oidx, optr[1:-1].astype(np.int64))
    assert all(len(a) == LEN for a in lists[STEP:2 * STEP])
    want = O.tri_count(optr, oidx)
    assert want == _triangles()
    with gb.Graph.upload(ptr, idx, n) as g:
        p, i, perm = g.download()
        assert np.array_equal(perm, np.arange(n))  # ranks follow ids
        v = i[int(p[STEP]):int(p[STEP + 1])].astype(np.int64)  # N+(v_0)
        assert len(v) == LEN and np.all(np.diff(v) == STEP)
        assert g.count() == want


@pytest.mark.parametrize("n", [0xFFFF << 10, (0xFFFF << 10) + 1])  # the last size with pair sets, the first without
def test_ids_of_more_than_26_bits(cuda, n):
    """The same graph in the last ids of n; isolated vertices rank below it."""
    import torch

    src, dst, m = _colliding()
    off = n - m
    s, d = (torch.from_numpy((x.astype(np.int64) + off).astype(np.int32)).cuda() for x in (src, dst))
    with gb.csr_from_edges_device(s, d, n) as c:
        nnz = c.shape()[1]

        class _Array:
            def __init__(self, ptr, count, typestr):
                self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}

        p, i = c.device_ptrs()
        with gb.Graph.upload(torch.as_tensor(_Array(p, n + 1, "<i8"), device="cuda"),
                             torch.as_tensor(_Array(i, nnz, "<i4"), device="cuda"), n) as g:
            assert g.count() == _triangles()
