"""Batches near the frame limit: which threads clear a launch's tables.

k_reduce runs gx x frames x 2 blocks of 256 threads, gx up to four an SM, and
clears the bin, segment and histogram tables beside its reductions.  With many
frames that grid has more threads than an int numbers, so the share of a thread
is a rule of its own (clear_share): every entry cleared once, and no index or
index plus stride beyond an int, at the largest shapes that a launch accepts.
"""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include "fdzb_internal.h"
#include <cstdio>
#include <vector>
using namespace fdzb;

// every entry of a table of n cleared exactly once
static bool once(int gx, int frames, int sm, int n)
{
    std::vector<int> seen(n, 0);
    const int blocks = clear_blocks(gx, frames, sm);
    int zero = 0;
    for (int z = 0; z < 2; ++z)
        for (int y = 0; y < frames; ++y)
            for (int x = 0; x < gx; ++x)
                for (int t = 0; t < 256; ++t) {
                    const ClearShare s = clear_share(blocks, x, y, z, gx, 256, t);
                    zero += s.first == 0;
                    if (s.first >= 0)
                        for (int i = s.first; i < n; i += s.stride) ++seen[i];
                }
    for (int v : seen)
        if (v != 1) return false;
    return zero == 1;
}

// the shares of a grid too large to walk: the last thread of the last block that
// clears, the first that does not, and the grid's last
static bool bounded(int gx, int frames, int sm, long long entries)
{
    const int blocks = clear_blocks(gx, frames, sm);
    auto at = [&](long long block, int t) {
        return clear_share(blocks, (unsigned)(block % gx), (unsigned)(block / gx), 1, gx, 256, t);
    };
    const ClearShare last = at(blocks - 1, 255);
    if (last.first != blocks * 256 - 1 || last.stride != blocks * 256) return false;
    if (entries + last.stride > 0x7fffffffll) return false;
    const long long all = (long long)gx * frames;
    for (long long b : {(long long)blocks, all / 2, all - 1})
        if (b >= blocks && b < all && at(b, 0).first >= 0) return false;
    return clear_share(blocks, 0, 0, 0, gx, 256, 0).first < 0;
}

int main()
{
    const long long bins = (1ll << 27) + 1;   // the most bins of a launch, and the unbinned slot
    bool ok = true;
    for (int gx : {1, 3, 64, 592})
        for (int frames : {1, 2, 7, 40})
            for (int n : {1, 64, 3072, 70001}) ok = ok && once(gx, frames, gx == 64 ? 2 : 148, n);
    for (int gx : {1, 64, 256, 592})
        for (int frames : {1, 7085, 7086, 16384, 65535}) ok = ok && bounded(gx, frames, 148, bins);
    std::puts(ok ? "ok" : "wrong");
    return ok ? 0 : 1;
}
"""


def test_the_clearing_share_of_a_grid_covers_every_entry_once_within_an_int(tmp_path):
    src = tmp_path / "share.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "share"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["/usr/bin/g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "4dzb_b200", "csrc"), "-I",
                    os.path.join(cuda, "include"), str(src), "-o", str(exe)], check=True, capture_output=True, text=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout.strip() == "ok"


@pytest.mark.gpu
@pytest.mark.parametrize("frames,vertices", [(6000, 0), (16384, 65537)])
def test_thousands_of_frames_equal_one(cuda_ok, fdzb, scenes, frames, vertices):
    """One small scene as every frame of a batch; with a vertex buffer of 65,537
    (most of them copies that no triangle names) k_reduce's grid has 2^31 threads."""
    import torch
    s = scenes.make_scene(8, 8, 5, n=4, bins=4, seed=7, sigma=0.8)
    pad = max(0, vertices - s.V)
    s.vtx = np.concatenate([s.vtx, np.repeat(s.vtx[:1], pad, axis=0)])
    pos, nrm, vtx, idx = fdzb.upload_scene(s)
    ctx, t = fdzb.context_for_scene(s, masks=True)
    ctx.launch()
    want = t["shadow"].clone(), t["masks"].clone()
    ctx.close()
    shadow = torch.full((frames, s.S), -1.0, device="cuda")
    masks = torch.full((frames, s.S * fdzb.mask_words(4)), -1, device="cuda", dtype=torch.int32)
    b = fdzb.Batch()
    desc = [fdzb.frame_desc(pos, nrm, s.W, s.H, vtx, s.V, idx, s.T, s.light, shadow[k], masks[k], bins=s.bins,
                            cull=s.cull, esp=s.esp) for k in range(frames)]
    for _ in range(2):
        shadow.fill_(-1.0)
        masks.fill_(-1)
        torch.cuda.synchronize()   # the batch has a stream of its own
        b.launch(desc)
        assert torch.equal(shadow.view(torch.int32), want[0].view(torch.int32).reshape(1, -1).expand(frames, -1))
        assert torch.equal(masks, want[1].reshape(1, -1).expand(frames, -1))
    b.close()
    assert (want[0] > 0).any()
