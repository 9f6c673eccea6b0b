"""Small launches, where a block's warps share an item: at the edges of the chunk split, against the oracle.

The warps of a block take a chunk of the bin's triangles each in turn; lists are
shorter than the warps, end inside a chunk or span several rounds; items hold 32
or 128 samples; grids use each row word; a pair limit splits the triangles into
passes that add to one another's masks.  The counting form runs a warp per item
and must give the same results, as must a launch with more items than blocks.
"""
import dataclasses

import pytest

import oracle
from tests import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,T,rows,cols,bins,chunk,item,limit", [
    (61, 37, 1, 8, 8, 1, 32, 32, 0),         # one triangle for four warps
    (61, 37, 3, 16, 16, 1, 32, 128, 0),
    (61, 37, 130, 16, 32, 2, 32, 32, 0),     # 32-row masks, a last chunk of few
    (61, 37, 700, 33, 33, 1, 8, 128, 0),     # 64-bit rows: a warp per block, no team
    (96, 60, 500, 8, 8, 8, 8, 32, 0),
    (96, 60, 4000, 17, 5, 8, 32, 64, 2000),   # several triangle passes
    (208, 150, 300, 8, 8, 8, 32, 32, 0),     # the two sides of the rule: 975 + 64 items at most
    (208, 149, 300, 8, 8, 8, 32, 32, 0),
])
@pytest.mark.parametrize("depth", [False, True])
def test_masks_equal_the_oracle(cuda_ok, fdzb, scenes, W, H, T, rows, cols, bins, chunk, item, limit, depth):
    s = scenes.make_scene(W, H, T, n=rows, bins=bins, seed=11, sigma=0.4)
    s = dataclasses.replace(s, light=dataclasses.replace(s.light, n=rows, nh=cols), depth_plane=depth)
    orc = oracle.frame(s)
    ctx, t = fdzb.context_for_scene(s, masks=True, tri_order=1)
    ctx.set_occlusion_shape(chunk, item)
    if limit:
        ctx.set_pair_capacity_limit(limit)
    for counting in (0, 1):
        ctx.set_profiling(counting)
        for k in ("shadow", "masks"):
            t[k].fill_(7)
        ctx.launch()
        errs = parity.compare(s, gpu=parity.collect(ctx, t, s, tri_order=1, intermediates=False), orc=orc)
        assert not errs, (counting, errs)
    assert (ctx.stats()["triangle_passes"] > 1) == bool(limit)
    ctx.close()
