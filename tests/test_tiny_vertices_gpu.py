"""Light middle vertices counted without a set (at most 16 higher neighbours):
out-degrees around one and two octets and past the limit, graphs of a few
vertices up to several tiles, and batches whose groups of 32 light vertices
cross graph borders.  Against the CPU oracle."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import gary_b200 as gb
from gary_b200 import _lib
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _circulant(n, k):
    """Every vertex joined to the next k ones (mod n): d+ = k but for the wrap."""
    v = np.repeat(np.arange(n), k)
    w = (v + np.tile(np.arange(1, k + 1), n)) % n
    return v.astype(np.uint32), w.astype(np.uint32)


@pytest.mark.parametrize("n", [40, 1000, 20011])
@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 15, 16, 17, 19])
def test_out_degrees_around_the_octets(cuda, n, k):
    src, dst = _circulant(n, k)
    ptr, idx = O.sym_csr(src, dst, n)
    optr, oidx = O.orient(ptr, idx)
    with gb.Graph.upload(ptr, idx, n) as g:
        assert g.count() == O.tri_count(optr, oidx)


@pytest.mark.parametrize("sizes", [[3, 4, 5] * 30, [5, 33, 31, 64, 7, 200, 3], [1, 2, 3, 1, 40]])
def test_batches_across_graph_borders(cuda, sizes):
    import torch

    rng = np.random.default_rng(len(sizes))
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    src, dst, want = [], [], []
    for n, o in zip(sizes, off[:-1]):
        s, d = rng.integers(0, n, 6 * n), rng.integers(0, n, 6 * n)
        ptr, idx = O.sym_csr(s.astype(np.uint32), d.astype(np.uint32), n)
        want.append(O.tri_count(*O.orient(ptr, idx)))
        src.append(s + int(o)), dst.append(d + int(o))
    n = int(off[-1])
    ptr, idx = O.sym_csr(np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32), n)
    h = C.c_void_p()
    L = gb.load()
    _lib.check(L.gary_batch_upload(off.ctypes.data, len(sizes), ptr.ctypes.data, idx.ctypes.data, n, len(idx), 0, None,
                                   C.byref(h)), "gary_batch_upload")
    g = gb.Graph(h.value)
    counts = torch.zeros(len(sizes), dtype=torch.int64, device="cuda")
    total = torch.zeros(1, dtype=torch.int64, device="cuda")
    _lib.check(L.gary_batch_count_async(g.handle, 0, counts.data_ptr(), total.data_ptr(), None), "gary_batch_count_async")
    assert counts.cpu().tolist() == want and int(total.item()) == sum(want)
    g.free()
