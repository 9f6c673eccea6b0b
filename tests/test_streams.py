"""Launches on a caller's stream, among the caller's own work on it.

A launch forks to a stream of its own for the sorts and joins before the occlusion
stage; the caller's stream has to see none of that: inputs written on it just
before a launch are read, outputs are complete for what follows on it, and inputs
may be overwritten there right away (once the pair buffer holds the launch's pairs).  On streams the caller made, the legacy
default stream and the per-thread default stream; with graphs, eagerly, and under
a capture of the caller's; two threads with a context each.
"""
import ctypes
import importlib
import os
import threading

import pytest

pytestmark = pytest.mark.gpu
scenes = importlib.import_module("4dzb_b200.scenes")
CASES = [(200, 150, 3000, 16, 16), (61, 37, 130, 8, 4)]     # a warp an item, a block an item


def _scene(W, H, T, n, bins, seed):
    return scenes.make_scene(W, H, T, n=n, bins=bins, seed=seed, sigma=0.3)


def _want(fdzb, ss):
    out = []
    for s in ss:
        ctx, t = fdzb.context_for_scene(s, masks=True)
        ctx.launch()
        out.append((t["shadow"].clone(), t["masks"].clone()))
        ctx.close()
    return out


def _handle(fdzb, kind, s, t):
    """(set_stream, set_graph, launch_async, sync, close) of a context or a batch on tensors t."""
    if kind == "ctx":
        ctx = fdzb.Context()
        ctx.set_view(s.W, s.H)
        ctx.set_bin_num(s.bins)
        ctx.set_scenes_esp(s.esp)
        ctx.set_backface_cull(s.cull)
        ctx.add_model(t["vtx"], s.V, 16, t["idx"], s.T, "scene")
        ctx.set_sample_buffers(t["pos"], t["nrm"])
        ctx.set_output_buffer(t["shadow"], t["masks"])
        ctx.set_area_light(s.light)
        return ctx.set_stream, ctx.set_graph, ctx.launch_async, ctx.sync, ctx.close
    b = fdzb.Batch()
    d = [fdzb.frame_desc(t["pos"], t["nrm"], s.W, s.H, t["vtx"], s.V, t["idx"], s.T, s.light, t["shadow"], t["masks"],
                         bins=s.bins, cull=s.cull, esp=s.esp)]
    return b.set_stream, b.set_graph, lambda: b.launch_async(d), b.sync, b.close


def _tensors(fdzb, s):
    import torch
    pos, nrm, vtx, idx = fdzb.upload_scene(s)
    return dict(pos=pos, nrm=nrm, vtx=vtx, idx=idx, shadow=torch.zeros(s.S, device="cuda"),
                masks=torch.zeros(s.S * fdzb.mask_words(s.light.n), dtype=torch.int32, device="cuda"))


@pytest.mark.parametrize("shape", CASES)
@pytest.mark.parametrize("kind", ["ctx", "batch"])
@pytest.mark.parametrize("stream", ["made", "legacy", "per-thread"])
@pytest.mark.parametrize("graph", [True, False])
def test_launches_are_ordered_with_the_callers_work(cuda_ok, fdzb, shape, kind, stream, graph):
    import torch
    ss = [_scene(*shape, seed=k) for k in (1, 2)]
    want, src = _want(fdzb, ss), [_tensors(fdzb, s) for s in ss]
    t = _tensors(fdzb, ss[0])
    st = {"made": torch.cuda.Stream, "legacy": torch.cuda.default_stream,
          "per-thread": lambda: torch.cuda.ExternalStream(2)}[stream]()
    set_stream, set_graph, launch_async, sync, close = _handle(fdzb, kind, ss[0], t)
    set_stream(1 if stream == "legacy" else st.cuda_stream)
    set_graph(graph)
    for k in (0, 1):      # grows the pair buffer: a launch that overflows it runs again in the sync
        for name in ("pos", "nrm", "vtx"):
            t[name].copy_(src[k][name])
        torch.cuda.synchronize()
        launch_async()
        sync()
    got = []
    with torch.cuda.stream(st):
        for k in (0, 1, 1, 0):
            torch.cuda._sleep(1_000_000)               # the launch is queued behind the copies
            for name in ("pos", "nrm", "vtx"):
                t[name].copy_(src[k][name])
            t["shadow"].fill_(-1.0)
            t["masks"].fill_(-1)
            launch_async()
            got.append((k, t["shadow"].clone(), t["masks"].clone()))
            for name in ("pos", "nrm", "vtx"):
                t[name].fill_(float("nan"))
        sync()
    torch.cuda.synchronize()
    for k, shadow, masks in got:
        assert torch.equal(shadow.view(torch.int32), want[k][0].view(torch.int32))
        assert torch.equal(masks, want[k][1])
    close()


@pytest.mark.parametrize("shape", CASES)
def test_a_launch_in_a_callers_capture(cuda_ok, fdzb, shape):
    import torch
    rt = ctypes.CDLL(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so.12"))
    vp = ctypes.c_void_p
    ss = [_scene(*shape, seed=k) for k in (1, 2)]
    want, src = _want(fdzb, ss), [_tensors(fdzb, s) for s in ss]
    t = _tensors(fdzb, ss[0])
    st = torch.cuda.Stream()
    set_stream, set_graph, launch_async, sync, close = _handle(fdzb, "ctx", ss[0], t)
    set_stream(st.cuda_stream)
    set_graph(False)
    for k in (0, 1):                                   # its buffers are there, and large enough
        for name in ("pos", "nrm", "vtx"):
            t[name].copy_(src[k][name])
        torch.cuda.synchronize()
        launch_async()
        sync()
    assert rt.cudaStreamBeginCapture(vp(st.cuda_stream), ctypes.c_int(2)) == 0
    launch_async()
    graph, run = vp(), vp()
    assert rt.cudaStreamEndCapture(vp(st.cuda_stream), ctypes.byref(graph)) == 0
    assert rt.cudaGraphInstantiate(ctypes.byref(run), graph, ctypes.c_ulonglong(0)) == 0
    for k in (1, 0, 1):
        with torch.cuda.stream(st):
            for name in ("pos", "nrm", "vtx"):
                t[name].copy_(src[k][name])
            t["shadow"].fill_(-1.0)
            t["masks"].fill_(-1)
            assert rt.cudaGraphLaunch(run, vp(st.cuda_stream)) == 0
        st.synchronize()
        assert torch.equal(t["shadow"].view(torch.int32), want[k][0].view(torch.int32))
        assert torch.equal(t["masks"], want[k][1])
    rt.cudaGraphExecDestroy(run)
    rt.cudaGraphDestroy(graph)
    close()


def test_two_threads_with_a_context_each(cuda_ok, fdzb):
    import torch
    ss = [_scene(*shape, seed=5) for shape in CASES]
    want, ts = _want(fdzb, ss), [_tensors(fdzb, s) for s in ss]
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        try:
            _, _, launch_async, sync, close = _handle(fdzb, "ctx", ss[k], ts[k])
            for _ in range(30):
                launch_async()
                sync()
                if not (torch.equal(ts[k]["shadow"], want[k][0]) and torch.equal(ts[k]["masks"], want[k][1])):
                    wrong.append(k)
            close()
        except Exception as e:   # noqa: BLE001
            wrong.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not wrong
