"""Profiling a graph that has been counted takes no second plan where the
counting plan has no hub rows, and the same cycles' worth of features either way."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from gary_b200 import costmodel as cm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rmat", [False, True])  # without and with hub rows
def test_profile_after_a_count(cuda, rmat):
    import torch

    n = 1 << 17
    src, dst = gb.gen_rmat(17, 2, 16 << 17) if rmat else gb.gen_er(n, 16 * n, 2)
    ptr, idx = gb.csr_from_edges(src, dst, n)
    lib = gb.load()
    try:
        lib.gary_tune(b"pool_keep_bytes", 0)
        with gb.Graph.upload(ptr, idx, n) as g:
            x0, legal0, _, c0 = cm.profile(g, variants=(-1,))
        with gb.Graph.upload(ptr, idx, n) as g:
            want = g.count()
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            x = torch.empty((n, 6), dtype=torch.float32, device="cuda")
            legal = torch.empty(n, dtype=torch.uint8, device="cuda")
            held = free - torch.cuda.mem_get_info()[0]  # by these two
            gb._lib.check(lib.gary_tc_features(g.handle, x.data_ptr(), legal.data_ptr(), None), "features")
            torch.cuda.synchronize()
            plan = free - torch.cuda.mem_get_info()[0] - held
            assert c0 == want
            assert np.array_equal(x.cpu().numpy(), x0) and np.array_equal(legal.cpu().numpy(), legal0)
            if not rmat:
                assert plan < 4 << 20, plan  # a plan holds 8 bytes for each of 2 M edges
    finally:
        lib.gary_tune(b"pool_keep_bytes", (1 << 64) - 1)
