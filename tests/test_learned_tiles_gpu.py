"""Tiles of learned plans: costs, tile targets and the least size of a split
vertex's pieces are all in predicted cycles.  Under a model that predicts one
cycle for every vertex the costs are the plain plan's probe counts in another
unit, so the tiles are the plain plan's."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from gary_b200 import _lib
from gary_b200 import costmodel as cm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,ef", [(14, 16), (16, 16), (18, 16)])
@pytest.mark.parametrize("tile_cost", [1024, 2048, 4096])  # a tile of the model holds 4096 cycles at least
def test_tiles_do_not_depend_on_the_unit_of_cost(cuda, scale, ef, tile_cost):
    src, dst = gb.gen_rmat(scale, scale, ef << scale)
    ptr, idx = gb.csr_from_edges(src, dst, 1 << scale)
    p = np.zeros(cm.n_params(), np.float32)
    p[6:12] = p[16:20] = 1  # standard deviations of inputs and outputs
    try:
        _lib.check(_lib.load().gary_tune(b"warp_tile_cost", tile_cost), "warp_tile_cost")
        cm.CostModel(p).install()
        with gb.Graph.upload(ptr, idx, 1 << scale) as g:
            want = g.count()
            plain = g.last_stats()
            assert g.count(sched=_lib.GARY_SCHED_LEARNED) == want
            learned = g.last_stats()
        assert learned["tiles"] == plain["tiles"]
        assert learned["cta_tiles"] == plain["cta_tiles"]
    finally:
        _lib.load().gary_tune(b"reset", 0)
        _lib.load().gary_set_cost_model(None)
