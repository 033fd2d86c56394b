"""4-cycles of sparse graphs: the light vertices a warp claims at a time go from
1 to 32 with their number.  Against the CPU oracle."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 3000, 16000, 40001, 200000, 900001])
def test_four_cycles_of_sparse_graphs(cuda, n):
    rng = np.random.default_rng(n)
    m = 6 * n
    ptr, idx = O.sym_csr(rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32), n)
    with gb.Graph.upload(ptr, idx, n) as g:
        assert g.count(gb.GARY_PATTERN_4CYCLE) == O.c4_count(ptr, idx)
