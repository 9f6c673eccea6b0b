"""The rasteriser's tile lists and per-tile records at their edges, against the oracle.

Sub-triangles of up to four tiles take their list places when they are counted,
larger ones when the lists are filled; records within 1024 pixels are evaluated
in 32 bits, larger ones in 64; a draw whose lists outgrow their buffer (its
first size: six tiles a triangle and four a tile) reads the triangles' boxes
instead, and the next draw has a larger buffer.
"""
import importlib

import numpy as np
import pytest

from oracle import orc
from tests.test_raster import _dev, _draw, _same, _targets

pytestmark = pytest.mark.gpu
scenes = importlib.import_module("4dzb_b200.scenes")


@pytest.mark.parametrize("W,H,T,sigma,grid", [
    (640, 360, 4000, 0.02, 64),     # mostly one tile a triangle
    (640, 360, 800, 0.6, 4),        # four tiles and a few more
    (640, 360, 300, 5.0, 1),        # every list full of large triangles: the buffer overflows
    (2300, 40, 60, 5.0, 1),         # wider than 1024 pixels: 64-bit edge functions
    (1, 1, 50, 0.15, 2), (17, 33, 500, 0.15, 8),
])
def test_targets_equal_the_oracle(cuda_ok, fdzb, W, H, T, sigma, grid):
    ms = scenes.mesh_scene(W, H, grid=grid, T=T, sigma=sigma)
    dev, t = _dev(fdzb, ms), _targets(ms)
    o = orc.raster(ms.vtx, ms.idx, ms.materials, ms.model, ms.view_proj, W, H, tri_material=ms.tri_material)
    r = fdzb.Raster()
    for _ in range(2):              # the second draw finds a buffer of the first one's size
        for k in t:
            t[k].fill_(-7.0)
        _draw(fdzb, r, ms, t, dev, ms.T)
        assert r.stats()["sub_triangles"] == o["sub_tris"]
        for k in ("g0", "g1", "g2", "g3", "depth"):
            _same(t[k], o[k], k)
    r.close()
