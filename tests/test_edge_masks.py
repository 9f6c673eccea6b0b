"""The fast pair test of the edge-mask kernel at the sizes and shapes where it can go wrong.

k_occlusion takes a pair's row masks from the projected triangle wherever the
crossings stay clear of the integer columns by a bound on the reference's FP32
error, and from the reference's own operations elsewhere.  Both must give the
oracle's masks bit for bit: on lattices whose edges pass exactly through light
samples (every crossing an integer), on slivers and on triangles smaller than
the spacing of the light samples, on triangles that reach the samples' depth or
the light's plane, on triangles far larger than the light, and on grids at the
edges of the row words (16, 17, 31, 32, 33 and 64 rows or columns, single rows).
"""
import dataclasses

import numpy as np
import pytest

import oracle
from tests import parity

pytestmark = pytest.mark.gpu

KINDS = ["lattice", "sliver", "tiny", "huge", "straddling", "behind"]
GRIDS = [(16, 16), (5, 16), (16, 31), (16, 32), (17, 3), (32, 32), (33, 31), (64, 64), (1, 1)]


def shaped(scenes, kind, rows, cols, seed=3):
    s = scenes.make_scene(120, 75, 700, n=rows, bins=8, seed=seed, sigma=0.3)
    light = dataclasses.replace(s.light, n=rows, nh=cols)
    v = s.vtx[:, :3].astype(np.float64).reshape(-1, 3, 3)
    c = v.mean(axis=1, keepdims=True)
    pos = s.pos.copy()
    if kind == "lattice":
        # light samples, receivers and vertices on multiples of 1/16, heights that halve or quarter the way
        light = dataclasses.replace(light, right_radius=rows / 16.0, top_radius=cols / 16.0,
                                    position=((rows - 1) / 16.0, (cols - 1) / 16.0, 6.0))
        pos[:, :2] = np.round(pos[:, :2] * 16.0) / 16.0
        pos[:, 2] = 0.0
        v[..., :2] = np.round(v[..., :2] * 16.0) / 16.0
        v[..., 2] = np.where(v[..., 2] < 1.6, 1.5, 3.0)
    elif kind == "sliver":
        v = c + (v - c) * np.array([1.0, 1e-3, 1.0]) + np.array([[0.0, 0, 0], [1e-4, 0, 0], [0, 1e-4, 0]])
    elif kind == "tiny":
        v = c + (v - c) * 0.02
    elif kind == "huge":
        v = c + (v - c) * np.array([8.0, 8.0, 0.3])
    elif kind == "straddling":
        v[..., 2] -= 1.4
    elif kind == "behind":
        v[..., 2] += 3.0
    vtx = s.vtx.copy()
    vtx[:, :3] = v.reshape(-1, 3).astype(np.float32)
    return dataclasses.replace(s, vtx=vtx, pos=pos, light=light, depth_plane=kind == "behind")


@pytest.mark.parametrize("rows,cols", GRIDS)
@pytest.mark.parametrize("kind", KINDS)
def test_masks_equal_the_oracle(cuda_ok, fdzb, scenes, kind, rows, cols):
    s = shaped(scenes, kind, rows, cols)
    orc = oracle.frame(s)
    for mode in (fdzb.OPEN_BOX_OFF, fdzb.OPEN_BOX_ON):
        ctx, t = fdzb.context_for_scene(s, masks=True, tri_order=1)
        ctx.set_open_box(mode)
        ctx.launch()
        errs = parity.compare(s, gpu=parity.collect(ctx, t, s, tri_order=1, intermediates=False), orc=orc)
        ctx.close()
        assert not errs, (mode, errs)
    assert (orc.arrays["shadow"] > 0).any()
