"""Random scenes: the edge-mask kernel against the reference's test for every pair.

The lane-per-pair schedule takes every pair's masks from the reference's operations;
the default takes them from projected triangles where that is certain.  Both run on
scenes with tilted and off-centre lights, far from the origin, with triangles
edge-on to the light or a sample, repeated vertices, vertices at samples, samples close
under the light and triangles near the samples' level.
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = ["soup", "far", "tilted", "edge-on", "degenerate", "near", "level"]


def _scene(scenes, kind, r):
    n = int(r.choice([1, 3, 8, 16, 17, 32]))
    s = scenes.make_scene(int(r.integers(3, 260)), int(r.integers(3, 160)), int(np.exp(r.uniform(0, 8))), n=n,
                          bins=int(r.choice([1, 8, 16, 64])), seed=int(r.integers(1 << 30)), sigma=float(r.choice([0.05, 0.2, 0.6])))
    pos, T = s.pos.astype(np.float64), s.T
    v = s.vtx[:, :3].astype(np.float64).reshape(T, 3, 3)
    lpos, view, up = np.array([0.0, 0.0, 6.0]), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0)
    some = pos[r.integers(0, s.S, T), :3]
    some = np.where(np.isnan(some), 0.0, some)
    if kind == "far":
        o = r.choice([-1.0, 1.0], 3) * 10.0 ** r.uniform(0, 5, 3)
        pos[:, :3] += o
        v += o
        lpos = lpos + o
    elif kind == "tilted":
        a = r.uniform(0.2, 1.5)
        lpos = np.array([-r.uniform(2, 9), r.uniform(-1, 1), r.uniform(0.3, 5)])
        view, up = (np.sin(a), r.uniform(-0.2, 0.2), -np.cos(a)), (r.uniform(-0.2, 0.2), 1.0, r.uniform(-0.2, 0.2))
    elif kind == "edge-on":
        to = lpos + (r.random((T, 3)) - 0.5) * [2.0, 2.0, 0.0] - some
        v = some[:, None] + to[:, None] * r.random((T, 3, 1))
        v[:, 2] += r.normal(size=(T, 3)) * 10.0 ** r.uniform(-8, -1)
    elif kind == "degenerate":
        v[::3, 1] = v[::3, 0]
        v[1::5, 2] = v[1::5, 0] + r.normal(size=v[1::5, 0].shape) * 1e-6
        v[2::4, 0] = some[2::4]
    elif kind == "near":
        pos[:, 2] = 6.0 - 10.0 ** r.uniform(-5, 1, s.S)
        v[:, :, 2] = 6.0 - 10.0 ** (r.uniform(-5, 1, (T, 1)) + 0.1 * r.random((T, 3)))
        pos[:, :2] *= 0.2
        v[:, :, :2] *= 0.3
    elif kind == "level":
        pos[:, 2] = 0.0
        v[:, :, 2] = 10.0 ** r.uniform(-5, 0, (T, 1)) * (1.0 + r.random((T, 3)))
    vtx = s.vtx.copy()
    vtx[:, :3] = v.reshape(-1, 3)
    radius = float(r.choice([0.25, 1.0, 2.0]))
    light = dataclasses.replace(s.light, right_radius=radius, top_radius=float(r.choice([radius, 0.7])), view_dir=view,
                                up_dir=up, position=tuple(float(x) for x in lpos))
    return dataclasses.replace(s, pos=pos.astype(np.float32), vtx=vtx, light=light, esp=float(r.choice([0.0, 1e-3])))


@pytest.mark.parametrize("kind", KINDS)
def test_masks_equal_the_reference_test_for_every_pair(cuda_ok, fdzb, scenes, kind):
    r = np.random.default_rng(KINDS.index(kind))
    lit = 0
    for k in range(12):
        s = _scene(scenes, kind, r)
        ctx, t = fdzb.context_for_scene(s, masks=True)
        ctx.set_occlusion_schedule(fdzb.OCC_LANE_PER_PAIR)
        ctx.launch()
        want = t["masks"].clone(), t["shadow"].clone()
        lit += int(want[0].count_nonzero())
        ctx.set_occlusion_schedule(fdzb.OCC_LANE_PER_SAMPLE)
        for mode in (fdzb.OPEN_BOX_OFF, fdzb.OPEN_BOX_ON):
            ctx.set_open_box(mode)
            ctx.launch()
            assert (t["masks"] == want[0]).all() and (t["shadow"] == want[1]).all(), (k, mode, s.W, s.H, s.T, s.light)
        ctx.close()
    assert lit
