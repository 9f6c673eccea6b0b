"""The rasteriser's buffers where the device has no room to spare, on the CPU.

fdzb_raster.cu's host code is built against a stand-in for the CUDA runtime whose
allocations have a limit and whose kernels do nothing.  Buffers are allocated with a
quarter to spare, and without where that does not fit.
"""
import ctypes
import importlib
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <cstdlib>
#include <cstring>
#include <string>
#include <cuda_runtime.h>

extern "C" size_t fake_limit = ~(size_t)0, fake_largest = 0;   // bytes of one allocation
static int s_object;
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
    if (n > fake_limit) { *p = nullptr; return cudaErrorMemoryAllocation; }
    if (n > fake_largest) fake_largest = n;
    return (*p = std::malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "stand-in"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)&s_object; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c) { *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)&s_object; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)&s_object; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
// what the compiler's launch and registration stubs call
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
void **__cudaRegisterFatBinary(void *) { return (void **)&s_object; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
char __cudaInitModule(void **) { return 0; }
}
namespace fdzb {
int set_error(int code, const std::string &) { return code; }
}
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("raster")
    (tmp / "fake.cpp").write_text(FAKE)
    out = str(tmp / "libraster.so")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    env = {k: v for k, v in os.environ.items() if k not in ("CC", "CXX")}
    # -Bsymbolic: the stand-in, whatever runtime this process has loaded
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-Xcompiler", "-fPIC",
                        "-shared", "-cudart", "none", "-Xlinker", "-Bsymbolic", "-I", os.path.join(ROOT, "include"),
                        os.path.join(ROOT, "4dzb_b200", "csrc", "fdzb_raster.cu"), str(tmp / "fake.cpp"), "-o", out],
                       capture_output=True, text=True, env=env)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def test_a_draw_without_room_to_spare(library):
    m = importlib.import_module("4dzb_b200")
    limit, largest = (ctypes.c_size_t.in_dll(library, k) for k in ("fake_limit", "fake_largest"))
    vp = ctypes.c_void_p
    library.fdzb_raster_create.argtypes = [ctypes.POINTER(vp), ctypes.c_int]
    library.fdzb_raster_draw.argtypes = [vp, ctypes.POINTER(m.RasterDesc)]
    library.fdzb_raster_destroy.argtypes = [vp]
    mem = np.zeros(4096, np.float32)
    at = (mem.ctypes.data + 63) // 64 * 64
    eye = np.eye(4, dtype=np.float32)
    d = m.raster_desc(at, 3, at, 100_000, at, 1, eye, eye, 16, 16, at, at, None, None, at)

    def draw():
        h = vp()
        assert library.fdzb_raster_create(ctypes.byref(h), 0) == 0
        rc = library.fdzb_raster_draw(h, ctypes.byref(d))
        assert library.fdzb_raster_destroy(h) == 0
        return rc

    assert draw() == 0
    spare = largest.value                       # the triangles' records, a quarter to spare
    limit.value, largest.value = spare - 1, 0
    assert draw() == 0 and largest.value < spare
    limit.value = spare * 4 // 5 - (1 << 14)    # less than they need
    assert draw() == -4                         # FDZB_ERR_NO_MEMORY
