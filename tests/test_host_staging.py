"""Launches whose pinned staging or device arena cannot grow, on the CPU.

fdzb_api.cpp is built against a small stand-in for the CUDA runtime: device and
pinned memory are host memory, copies happen at once, the kernels do nothing, and
a pinned allocation can be made to fail.  A batch that needs more staging than
there is fails with an error; what the handle knew of the launch before can still
be read afterwards, frames beyond it are refused, and the next launch works.  An arena is
allocated with an eighth to spare, and without where that does not fit.
"""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <cstdlib>
#include <cstring>
#include "fdzb_internal.h"

extern "C" int fake_pinned_left = 1 << 30;   // pinned allocations until one fails
extern "C" size_t fake_device_limit = ~(size_t)0, fake_device_asked = 0;   // bytes of one allocation
static int s_object;

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
    if (n > fake_device_limit) { *p = nullptr; return cudaErrorMemoryAllocation; }
    fake_device_asked = n;
    return (*p = std::calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)   // cudaMallocHost of typed pointers
{
    if (fake_pinned_left-- <= 0) { *p = nullptr; return cudaErrorMemoryAllocation; }
    *p = std::malloc(n);
    std::memset(*p, 0x5a, n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "stand-in"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)&s_object; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)&s_object; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)&s_object; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
// not called here: no graphs, no pointer checks
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *, const void *) { return cudaErrorNotSupported; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
}

namespace fdzb {
// The kernels' stand-in: every frame is done, with its place in the list as its count.
cudaError_t run_pipeline(const DeviceBuffers &b, int, int, int, cudaStream_t, cudaEvent_t *, int *launches, const ForkStream *)
{
    for (int i = 0; i < b.nframes; ++i) {
        b.states[i].state = 2;
        b.states[i].nValidTris = 1;
        b.states[i].nValidSamples = 100 + i;
    }
    b.counters->pairCount = 7 * b.nframes;
    if (launches) *launches = 1;
    return cudaSuccess;
}
size_t sort_tiles(size_t keys) { return keys / 1024 + 1; }
int sort_passes_for(long long) { return 1; }
cudaError_t run_move_model(float *, int, int, const float *, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t measure_alu_rate(double *) { return cudaErrorNotSupported; }
cudaError_t check_division(unsigned long long, unsigned long long, unsigned long long *, unsigned long long *)
{
    return cudaErrorNotSupported;
}
}
"""

SETUP = r"""
import ctypes, importlib, json, sys
sys.path.insert(0, sys.argv[1])
m = importlib.import_module("4dzb_b200")
lib = ctypes.CDLL(sys.argv[2])
left = ctypes.c_int.in_dll(lib, "fake_pinned_left")
vp, P, i32 = ctypes.c_void_p, ctypes.POINTER, ctypes.c_int32
lib.fdzb_batch_create.argtypes = [P(vp), i32]
lib.fdzb_batch_set_graph.argtypes = [vp, i32]
lib.fdzb_batch_launch.argtypes = [vp, P(m.FrameDesc), i32, P(ctypes.c_float)]
lib.fdzb_batch_get_stats.argtypes = [vp, P(m.BatchStats)]
lib.fdzb_batch_get_frame_stats.argtypes = [vp, i32, P(m.FrameStats)]
lib.fdzb_batch_destroy.argtypes = [vp]
mem = (ctypes.c_float * 4096)()
at = (ctypes.addressof(mem) + 63) // 64 * 64

def frames(n, tris=1):
    light = importlib.import_module("4dzb_b200.scenes").Light(right_radius=1.0, top_radius=1.0, n=4)
    return (m.FrameDesc * n)(*[m.frame_desc(at, at, 4, 4, at, 3, at, tris, light, at, None, bins=4) for _ in range(n)])

def batch():
    b = vp()
    assert lib.fdzb_batch_create(ctypes.byref(b), 0) == 0
    assert lib.fdzb_batch_set_graph(b, 0) == 0
    return b

b, ms, out = batch(), ctypes.c_float(), []

def totals():
    s = m.BatchStats()
    return [lib.fdzb_batch_get_stats(b, ctypes.byref(s)), s.totals.num_pairs]

def frame(i):
    s = m.FrameStats()
    rc = lib.fdzb_batch_get_frame_stats(b, i, ctypes.byref(s))
    return [rc, s.valid_samples if rc == 0 else 0]

def launch(n, tris=1):
    return lib.fdzb_batch_launch(b, frames(n, tris), n, ctypes.byref(ms))
"""

STAGING = r"""
out.append([launch(2), totals(), frame(0), frame(1)])
for fails in (0, 1):             # the first block of the larger launch, then its second
    left.value = fails
    out.append([launch(3000) != 0, totals(), frame(0), frame(1), frame(2999)[0] != 0])
    left.value = 1 << 30
out.append([launch(2), totals(), frame(1)])
out.append([launch(3000), totals(), frame(2999)])
assert lib.fdzb_batch_destroy(b) == 0
print(json.dumps(out))
"""

ARENA = r"""
limit, asked = (ctypes.c_size_t.in_dll(lib, k) for k in ("fake_device_limit", "fake_device_asked"))
assert launch(1, 20000) == 0
spare = asked.value                       # the need and an eighth, whole megabytes
for limit.value in (spare - 1, spare * 8 // 9 - (2 << 20)):
    b = batch()
    out.append([launch(1, 20000), asked.value < spare])
print(json.dumps(out))
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("staging")
    (tmp / "fake.cpp").write_text(FAKE)
    csrc = os.path.join(ROOT, "4dzb_b200", "csrc")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    out = str(tmp / "libstaging.so")
    r = subprocess.run(["/usr/bin/g++", "-O1", "-g", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", csrc, "-I",
                        os.path.join(cuda, "include"), os.path.join(csrc, "fdzb_api.cpp"),
                        os.path.join(csrc, "fdzb_light.cpp"), str(tmp / "fake.cpp"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def _drive(library, tmp_path, steps):
    script = tmp_path / "drive.py"
    script.write_text(SETUP + steps)
    r = subprocess.run([sys.executable, str(script), ROOT, library], capture_output=True, text=True,
                       env=dict(os.environ, MALLOC_PERTURB_="165"))
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
    return json.loads(r.stdout)


def test_statistics_outlive_a_launch_without_staging(library, tmp_path):
    first, no_frames, no_states, again, large = _drive(library, tmp_path, STAGING)
    assert first == [0, [0, 14], [0, 100], [0, 101]]
    for failed in (no_frames, no_states):
        assert failed == [True, [0, 14], [0, 100], [0, 101], True]
    assert again == [0, [0, 14], [0, 101]]
    assert large == [0, [0, 21000], [0, 3099]]


def test_an_arena_without_room_to_spare(library, tmp_path):
    """The launch runs where its need fits and the spare eighth does not; below the need it is refused."""
    fits, refused = _drive(library, tmp_path, ARENA)
    assert fits == [0, True]
    assert refused[0] == -4   # FDZB_ERR_NO_MEMORY
