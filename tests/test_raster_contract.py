"""What a draw refuses, and the state it leaves: the count of (sub-triangle, tile) pairs
is known when the draw returns, so a draw beyond 2^31 pairs is refused by the draw
itself, a capturing stream is refused, and the handle draws on afterwards.
"""
import ctypes
import importlib
import os

import numpy as np
import pytest

from oracle import orc
from tests.test_raster import _dev, _draw, _same, _targets

pytestmark = pytest.mark.gpu
scenes = importlib.import_module("4dzb_b200.scenes")


def _still_draws(fdzb, r, ms):
    dev, t = _dev(fdzb, ms), _targets(ms)
    o = orc.raster(ms.vtx, ms.idx, ms.materials, ms.model, ms.view_proj, ms.W, ms.H, tri_material=ms.tri_material)
    _draw(fdzb, r, ms, t, dev, ms.T)
    assert r.stats()["sub_triangles"] == o["sub_tris"]
    for k in ("g0", "g1", "g2", "g3", "depth"):
        _same(t[k], o[k], k)


def test_more_than_2_31_pairs_are_refused_by_the_draw(cuda_ok, fdzb):
    """2,050 triangles over every tile of a 16384 x 16384 view (1,024 x 1,024 tiles)."""
    import torch
    small = scenes.mesh_scene(64, 48)
    r = fdzb.Raster()
    _still_draws(fdzb, r, small)
    W, T = 16384, 2050
    vtx = np.zeros((3, 8), np.float32)
    vtx[:, :3] = [[-1, -1, 0], [3, -1, 0], [-1, 3, 0]]     # the identity matrices: the whole window
    dv = torch.from_numpy(vtx).cuda()
    idx = torch.tensor([[0, 1, 2]] * T, device="cuda", dtype=torch.int32)
    mats = torch.from_numpy(small.materials).cuda()
    g = [torch.zeros(W * W, 4, device="cuda") for _ in range(2)]
    eye = np.eye(4, dtype=np.float32)
    d = fdzb.raster_desc(dv, 3, idx, T, mats, len(mats), eye, eye, W, W, g[0], g[1], None, None, None)
    with pytest.raises(fdzb.FdzbError, match="2\\^31"):
        r.draw(d)
    st = r.stats()
    assert st["triangles"] == T and st["sub_triangles"] == T and st["tile_pairs"] == T << 20
    r.sync()
    assert not g[0].any()                                  # nothing was drawn
    del g
    _still_draws(fdzb, r, small)
    r.close()


def test_a_capturing_stream_is_refused(cuda_ok, fdzb):
    import torch
    rt = ctypes.CDLL(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so.12"))
    for f in (rt.cudaStreamBeginCapture, rt.cudaStreamEndCapture, rt.cudaGraphDestroy):
        f.restype = ctypes.c_int
    ms = scenes.mesh_scene(64, 48)
    s = torch.cuda.Stream()
    r = fdzb.Raster()
    r.set_stream(s.cuda_stream)
    _still_draws(fdzb, r, ms)                              # its buffers are there
    dev, t = _dev(fdzb, ms), _targets(ms)
    torch.cuda.synchronize()
    assert rt.cudaStreamBeginCapture(ctypes.c_void_p(s.cuda_stream), ctypes.c_int(2)) == 0
    try:
        with pytest.raises(fdzb.FdzbError):
            _draw(fdzb, r, ms, t, dev, ms.T)
    finally:
        graph = ctypes.c_void_p()
        rt.cudaStreamEndCapture(ctypes.c_void_p(s.cuda_stream), ctypes.byref(graph))
        if graph.value:
            rt.cudaGraphDestroy(graph)
        rt.cudaGetLastError()
    _still_draws(fdzb, r, ms)
    r.close()
