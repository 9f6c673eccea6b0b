"""The forms of the edge-mask kernel that the launch's size picks, on shapes where the
fast pair test can go wrong, and vertices that are no numbers of its range.

A launch of at most 7 items an SM has a block's warps share an item, larger ones run
a warp an item; 32 x 32 bins on 120 x 75 samples (281 + 1024 items at most) are beyond
that line, 8 x 8 bins within it.  Vertices at infinity, NaN, far out of the fast
test's range or at the edge of it send their triangles to the reference's test.
"""
import dataclasses

import numpy as np
import pytest

import oracle
from tests import parity
from tests.test_edge_masks import KINDS, shaped

pytestmark = pytest.mark.gpu


def _check(fdzb, s):
    orc = oracle.frame(s)
    for mode in (fdzb.OPEN_BOX_OFF, fdzb.OPEN_BOX_ON):
        ctx, t = fdzb.context_for_scene(s, masks=True, tri_order=1)
        ctx.set_open_box(mode)
        ctx.launch()
        errs = parity.compare(s, gpu=parity.collect(ctx, t, s, tri_order=1, intermediates=False), orc=orc)
        ctx.close()
        assert not errs, (mode, errs)
    return orc


@pytest.mark.parametrize("rows,cols", [(16, 16), (5, 31), (16, 32), (32, 32)])
@pytest.mark.parametrize("kind", KINDS)
def test_a_warp_an_item_equals_the_oracle(cuda_ok, fdzb, scenes, kind, rows, cols):
    orc = _check(fdzb, dataclasses.replace(shaped(scenes, kind, rows, cols), bins=32))
    assert (orc.arrays["shadow"] > 0).any()


@pytest.mark.parametrize("bins", [8, 32])
@pytest.mark.parametrize("value", [1e7, 3e6, -1e30, 3e38, np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("depth", [False, True])
def test_vertices_beyond_the_fast_test(cuda_ok, fdzb, scenes, bins, value, depth):
    """One coordinate of a vertex of every seventh triangle; x and y only, so that the
    far plane, which every vertex's depth moves, stays where the scene is."""
    s = shaped(scenes, "straddling" if depth else "huge", 16, 16)
    vtx = s.vtx.copy()
    for k in range(0, s.T, 7):
        vtx[s.idx[k, k % 3], (k // 7) % 2] = value
    s = dataclasses.replace(s, vtx=vtx, bins=bins, depth_plane=depth)
    ctx, t = fdzb.context_for_scene(s, masks=True, tri_order=1)
    ctx.set_open_box(fdzb.OPEN_BOX_OFF)
    ctx.set_depth_plane(False)
    ctx.set_occlusion_schedule(fdzb.OCC_LANE_PER_PAIR)    # the reference's test for every pair
    ctx.launch()
    want = t["masks"].clone()
    ctx.set_occlusion_schedule(fdzb.OCC_LANE_PER_SAMPLE)
    for mode in (fdzb.OPEN_BOX_OFF, fdzb.OPEN_BOX_ON):
        ctx.set_open_box(mode)
        ctx.launch()
        assert (t["masks"] == want).all(), mode
    ctx.close()
    assert want.any()
    _check(fdzb, s)
