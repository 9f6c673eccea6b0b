// fdzb_raster.cu -- G-buffer rasteriser: the view samples' producer.
//
// Replaces the app's GL G-buffer pass (4DZB/Render/Render.cpp:390-431 and
// DrawModel :267-340 with the gatherData shaders, 4DZB/Resources/shader/
// gatherData.shv/.shf) so that meshes feed the shadow pipeline without a
// graphics stack.  Per vertex worldPos = model*(P,1), worldN = model*(N,0),
// clip = view_proj*(worldPos,1); per pixel the nearest fragment (GL_LESS,
// earlier triangle wins ties) writes g0 = (worldPos, Ks.r), g1 = (worldN,
// Ks.g), g2 = (Ka, Ks.b), g3 = (Kd, shininess), worldPos and worldN
// interpolated perspective-correctly.  The rules GL leaves open are fixed (and
// restated by the oracle, oracle/fdzb_raster_oracle.c): near-plane clipping in
// clip space, window coordinates snapped to 1/16 pixel, coverage at pixel
// centres by exact 64-bit edge functions with an ownership rule for centres on
// an edge, depth 0..1 per fragment.  Every float operation is an _rn
// intrinsic, so the result is the oracle's bit for bit.
//
// B200 layout: one thread per triangle sets up at most two sub-triangles (the
// near-plane clip of a triangle is a triangle or a quad) into 144-byte records
// at slots 2t and 2t+1, with the 16 x 16 pixel tiles their pixel boxes touch (8
// bytes a slot), and counts the tiles' lists; the lists are laid out (k_rs_lists)
// and filled (k_rs_scatter); one 256-thread block per tile resolves its pixels
// and writes each once, cleared or drawn.  The host waits once, for the length of
// all lists, while they are being laid out (fdzb_raster_draw).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>

#include "../../include/fdzb.h"
#include "fdzb_device.cuh"
#include "fdzb_internal.h"

namespace fdzb {
namespace {

constexpr int kTile = 16;              // pixels per tile side
constexpr int kRecF4 = 9;              // float4s per sub-triangle record
constexpr int kChunk = kTile * kTile;  // records staged per round, one a thread
constexpr float kMaxWindow = 67108864.0f;   // 2^26 pixels

struct RasterCounters {
    unsigned long long subTris, dropped, pairs, badIdx, badMat;
    unsigned long long next;   // end of the tile lists laid out so far
};

struct RasterMats {
    float model[16], viewProj[16];   // column-major
};

struct RVert {
    float c[4];
    float p[3], n[3];
};

__device__ __forceinline__ void mat_vec4(const float *m, const float v[4], float out[4])
{
#pragma unroll
    for (int r = 0; r < 4; ++r)
        out[r] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[r], v[0]), __fmul_rn(m[4 + r], v[1])),
                                     __fmul_rn(m[8 + r], v[2])),
                           __fmul_rn(m[12 + r], v[3]));
}

__device__ __forceinline__ float lerp_rn(float a, float b, float t) { return __fadd_rn(a, __fmul_rn(t, __fsub_rn(b, a))); }

__device__ __forceinline__ RVert lerp_vert(const RVert &a, const RVert &b, float t)
{
    RVert o;
#pragma unroll
    for (int k = 0; k < 4; ++k) o.c[k] = lerp_rn(a.c[k], b.c[k], t);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        o.p[k] = lerp_rn(a.p[k], b.p[k], t);
        o.n[k] = lerp_rn(a.n[k], b.n[k], t);
    }
    return o;
}

struct SubTri {
    int X[3], Y[3];
    long long area;
    float z[3], iw[3];
    float p[3][3], n[3][3];
};

// Window setup of one sub-triangle; returns 1 if it can draw (non-zero area,
// every vertex in front and inside the 2^26-pixel window range), 2 if dropped.
__device__ int setup_sub(const RVert &a, const RVert &b, const RVert &c, int W, int H, SubTri &o)
{
    const RVert *v[3] = {&a, &b, &c};
    const float hw = __fmul_rn(0.5f, (float)W), hh = __fmul_rn(0.5f, (float)H);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float w = v[i]->c[3];
        if (!(w > 0.0f)) return 0;
        const float xn = __fdiv_rn(v[i]->c[0], w), yn = __fdiv_rn(v[i]->c[1], w), zn = __fdiv_rn(v[i]->c[2], w);
        const float xw = __fadd_rn(__fmul_rn(xn, hw), hw), yw = __fadd_rn(__fmul_rn(yn, hh), hh);
        if (!(fabsf(xw) < kMaxWindow && fabsf(yw) < kMaxWindow)) return 2;
        o.X[i] = (int)__float2ll_rn(__fmul_rn(xw, 16.0f));
        o.Y[i] = (int)__float2ll_rn(__fmul_rn(yw, 16.0f));
        o.z[i] = __fadd_rn(__fmul_rn(zn, 0.5f), 0.5f);
        o.iw[i] = __fdiv_rn(1.0f, w);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            o.p[i][k] = v[i]->p[k];
            o.n[i][k] = v[i]->n[k];
        }
    }
    long long area = (long long)(o.X[1] - o.X[0]) * (long long)(o.Y[2] - o.Y[0]) -
                     (long long)(o.Y[1] - o.Y[0]) * (long long)(o.X[2] - o.X[0]);
    if (area == 0) return 0;
    if (area < 0) {   // counter-clockwise: swap vertices 1 and 2
        int t = o.X[1]; o.X[1] = o.X[2]; o.X[2] = t;
        t = o.Y[1]; o.Y[1] = o.Y[2]; o.Y[2] = t;
        float f = o.z[1]; o.z[1] = o.z[2]; o.z[2] = f;
        f = o.iw[1]; o.iw[1] = o.iw[2]; o.iw[2] = f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            f = o.p[1][k]; o.p[1][k] = o.p[2][k]; o.p[2][k] = f;
            f = o.n[1][k]; o.n[1][k] = o.n[2][k]; o.n[2][k] = f;
        }
        area = -area;
    }
    o.area = area;
    return 1;
}

// Pixel-centre box of a sub-triangle, clamped to the viewport (x0 > x1: none).
__device__ __forceinline__ void pixel_box(const int *X, const int *Y, int W, int H, int &x0, int &x1, int &y0,
                                          int &y1)
{
    const int mnx = min(X[0], min(X[1], X[2])), mxx = max(X[0], max(X[1], X[2]));
    const int mny = min(Y[0], min(Y[1], Y[2])), mxy = max(Y[0], max(Y[1], Y[2]));
    // centres x*16 + 8 inside [mnx, mxx]
    x0 = max((mnx - 8 + 15) >> 4, 0);
    x1 = min((mxx - 8) >> 4, W - 1);
    y0 = max((mny - 8 + 15) >> 4, 0);
    y1 = min((mxy - 8) >> 4, H - 1);
}

__device__ __forceinline__ void store_record(float4 *rec, const SubTri &s, int mat)
{
    rec[0] = make_float4(__int_as_float(s.X[0]), __int_as_float(s.Y[0]), __int_as_float(s.X[1]),
                         __int_as_float(s.Y[1]));
    rec[1] = make_float4(__int_as_float(s.X[2]), __int_as_float(s.Y[2]), __int_as_float((int)(s.area & 0xffffffffll)),
                         __int_as_float((int)(s.area >> 32)));
    rec[2] = make_float4(s.z[0], s.z[1], s.z[2], s.iw[0]);
    rec[3] = make_float4(s.iw[1], s.iw[2], __int_as_float(mat), 0.0f);
    rec[4] = make_float4(s.p[0][0], s.p[0][1], s.p[0][2], s.p[1][0]);
    rec[5] = make_float4(s.p[1][1], s.p[1][2], s.p[2][0], s.p[2][1]);
    rec[6] = make_float4(s.p[2][2], s.n[0][0], s.n[0][1], s.n[0][2]);
    rec[7] = make_float4(s.n[1][0], s.n[1][1], s.n[1][2], s.n[2][0]);
    rec[8] = make_float4(s.n[2][1], s.n[2][2], 0.0f, 0.0f);
}

// First and last tile columns and rows of a sub-triangle's pixel box, 16 bits
// each; a slot that draws nothing holds (first > last).
__device__ __forceinline__ uint2 tile_box(const SubTri &s, int W, int H)
{
    int x0, x1, y0, y1;
    pixel_box(s.X, s.Y, W, H, x0, x1, y0, y1);
    if (x0 > x1 || y0 > y1) return make_uint2(1u, 1u);
    return make_uint2((uint32_t)(x0 / kTile) | (uint32_t)(x1 / kTile) << 16,
                      (uint32_t)(y0 / kTile) | (uint32_t)(y1 / kTile) << 16);
}

__device__ __forceinline__ int box_tiles(uint2 b)
{
    const int w = (int)(b.x >> 16) - (int)(b.x & 0xffffu) + 1;
    return w > 0 ? w * ((int)(b.y >> 16) - (int)(b.y & 0xffffu) + 1) : 0;
}

// Calls f(k, tile) for tiles first..first + 3 of a box, row by row.
template <class F> __device__ __forceinline__ void four_tiles(uint2 b, int first, int n, int tilesX, F f)
{
    const int x0 = (int)(b.x & 0xffffu), w = (int)(b.x >> 16) - x0 + 1, y0 = (int)(b.y & 0xffffu);
    int y = first / w, x = first - y * w;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (first + k < n) f(k, (y0 + y) * tilesX + x0 + x);
        if (++x == w) {
            x = 0;
            ++y;
        }
    }
}

// Counts a slot's tiles.  The tiles of a box of at most four (most of them) are
// counted with their answer, the slot's place in the tile's list, which saves
// the scatter its own atomics; larger boxes only raise the tile's second count.
__device__ __forceinline__ void count_tiles(uint2 b, int tilesX, int *tileCount, int *tileMore, uint4 *__restrict__ place,
                                            unsigned long long &pairs)
{
    const int n = box_tiles(b);
    pairs += (unsigned long long)n;
    if (n > 4) {
        for (int k0 = 0; k0 < n; k0 += 4)
            four_tiles(b, k0, n, tilesX, [&](int, int tile) { atomicAdd(&tileMore[tile], 1); });
    } else if (n > 0) {
        uint32_t at[4] = {0u, 0u, 0u, 0u};
        four_tiles(b, 0, n, tilesX, [&](int k, int tile) { at[k] = (uint32_t)atomicAdd(&tileCount[tile], 1); });
        *place = make_uint4(at[0], at[1], at[2], at[3]);
    }
}

__global__ void k_rs_clear(int S, float4 *g0, float4 *g1, float4 *g2, float4 *g3, float *depth)
{
    const float nan = __int_as_float(0x7fc00000);
    const float4 q = make_float4(nan, nan, nan, nan);
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < S; p += gridDim.x * blockDim.x) {
        g0[p] = q;
        g1[p] = q;
        if (g2) g2[p] = q;
        if (g3) g3[p] = q;
        if (depth) depth[p] = 1.0f;
    }
}

// The near-plane case (z >= -w, Sutherland-Hodgman), out of line: the polygon's
// vertices are indexed and would put every triangle's in local memory.
__device__ __noinline__ int clip_near(const RVert v[3], RVert poly[4])
{
    int np = 0;
    for (int i = 0; i < 3; ++i) {
        const RVert &a = v[i], &b = v[(i + 1) % 3];
        const float da = __fadd_rn(a.c[2], a.c[3]), db = __fadd_rn(b.c[2], b.c[3]);
        if (da >= 0.0f) poly[np++] = a;
        if ((da >= 0.0f) != (db >= 0.0f)) poly[np++] = lerp_vert(a, b, __fdiv_rn(da, __fsub_rn(da, db)));
    }
    return np;
}

// One thread per triangle.  WIDE: vertices of 32 bytes, 16-byte aligned, with
// the position first and the normal at float 5 (the MeshManager layout), read
// as two 16-byte loads.  The counters are summed per block before they reach
// memory, and a triangle wholly in front of the near plane never touches local
// memory (1920 x 1080, 331k triangles: 408 -> 47 us; bound by the scattered
// vertex reads and the tile counts' atomics).
template <int WIDE>
__global__ void __launch_bounds__(128) k_rs_setup(const float *__restrict__ vtx, int V, int strideF, int posOff,
                                                  int nrmOff, const uint32_t *__restrict__ idx, int T,
                                                  const int32_t *__restrict__ triMat, int nMat,
                                                  const __grid_constant__ RasterMats mats, int W, int H, int tilesX,
                                                  float4 *__restrict__ recs, uint2 *__restrict__ boxes,
                                                  uint4 *__restrict__ places, int *__restrict__ tileCount,
                                                  int *__restrict__ tileMore, RasterCounters *ctr)
{
    __shared__ unsigned long long sCount[5];
    if (threadIdx.x < 5) sCount[threadIdx.x] = 0;
    __syncthreads();
    unsigned long long nsub = 0, ndrop = 0, npairs = 0, nbadI = 0, nbadM = 0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
        float4 *r0 = recs + (size_t)kRecF4 * (2 * (size_t)t);
        uint2 box0 = make_uint2(1u, 1u), box1 = box0;
        RVert v[3];
        bool ok = true, front = true;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const uint32_t id = idx[3 * (size_t)t + i];
            if (id >= (uint32_t)V) {
                ok = false;
                break;
            }
            const float *src = vtx + (size_t)id * strideF;
            float P[4], N[4];
            if (WIDE) {
                const float4 a = __ldg(reinterpret_cast<const float4 *>(src)), b = __ldg(reinterpret_cast<const float4 *>(src) + 1);
                P[0] = a.x, P[1] = a.y, P[2] = a.z;
                N[0] = b.y, N[1] = b.z, N[2] = b.w;
            } else {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    P[k] = src[posOff + k];
                    N[k] = src[nrmOff + k];
                }
            }
            P[3] = 1.0f;
            N[3] = 0.0f;
            float wp[4], wn[4];
            mat_vec4(mats.model, P, wp);
            mat_vec4(mats.model, N, wn);
            const float WP[4] = {wp[0], wp[1], wp[2], 1.0f};
            mat_vec4(mats.viewProj, WP, v[i].c);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                v[i].p[k] = wp[k];
                v[i].n[k] = wn[k];
            }
            front = front && __fadd_rn(v[i].c[2], v[i].c[3]) >= 0.0f;
        }
        if (!ok) {
            ++nbadI;
        } else {
            int mat = triMat ? triMat[t] : 0;
            if (mat < 0 || mat >= nMat) {
                ++nbadM;
                mat = 0;
            }
            SubTri s;
            if (front) {
                const int rc = setup_sub(v[0], v[1], v[2], W, H, s);
                if (rc == 2) ++ndrop;
                if (rc == 1) {
                    store_record(r0, s, mat);
                    ++nsub;
                    box0 = tile_box(s, W, H);
                }
            } else {
                RVert in[3] = {v[0], v[1], v[2]}, poly[4];
                const int np = clip_near(in, poly);
                for (int k = 0; k < np - 2; ++k) {   // triangle, or quad as two
                    const int rc = setup_sub(poly[0], poly[k + 1], poly[k + 2], W, H, s);
                    if (rc == 2) ++ndrop;
                    if (rc == 1) {
                        store_record(r0 + k * kRecF4, s, mat);
                        ++nsub;
                        (k ? box1 : box0) = tile_box(s, W, H);
                    }
                }
            }
            count_tiles(box0, tilesX, tileCount, tileMore, places + 2 * (size_t)t, npairs);
            if (!front) count_tiles(box1, tilesX, tileCount, tileMore, places + 2 * (size_t)t + 1, npairs);
        }
        reinterpret_cast<uint4 *>(boxes)[t] = make_uint4(box0.x, box0.y, box1.x, box1.y);
    }
    unsigned long long c[5] = {nsub, ndrop, npairs, nbadI, nbadM};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c[k] += __shfl_xor_sync(kFullWarp, c[k], o);
        if ((threadIdx.x & 31) == 0 && c[k]) atomicAdd(&sCount[k], c[k]);
    }
    __syncthreads();
    if (threadIdx.x < 5 && sCount[threadIdx.x]) {
        unsigned long long *dst[5] = {&ctr->subTris, &ctr->dropped, &ctr->pairs, &ctr->badIdx, &ctr->badMat};
        atomicAdd(dst[threadIdx.x], sCount[threadIdx.x]);
    }
}

// Lays the tiles' lists out end to end: a block's tiles by a scan of their
// counts, the blocks in the order in which they arrive (a list's place does not
// matter; 8,160 tiles: 3 us, 10 us as one block's scan of all tiles).  Hands the
// draw's counters to the host on the way (pinned memory).
__global__ void __launch_bounds__(256) k_rs_lists(const int *__restrict__ cnt, const int *__restrict__ more,
                                                  long long *__restrict__ start, int n, RasterCounters *ctr,
                                                  RasterCounters *host)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) *host = *ctr;   // k_rs_setup's are final
    __shared__ unsigned long long sWarp[8], sBase;
    const int i = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long c = i < n ? (unsigned long long)cnt[i] + (unsigned long long)more[i] : 0ull;
    unsigned long long x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(kFullWarp, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sWarp[warp] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long run = 0;
        for (int k = 0; k < 8; ++k) {
            const unsigned long long v = sWarp[k];
            sWarp[k] = run;
            run += v;
        }
        sBase = atomicAdd(&ctr->next, run);
    }
    __syncthreads();
    if (i < n) start[i] = (long long)(sBase + sWarp[warp] + x - c);
}

__global__ void k_rs_scatter(const uint4 *__restrict__ boxes, const uint4 *__restrict__ places, int T, int tilesX,
                             const int *__restrict__ tileCount, const long long *__restrict__ tileStart,
                             int *__restrict__ tileFill, int *__restrict__ pairs, long long capacity)
{
    auto put = [&](uint2 b, int slot) {
        const int n = box_tiles(b);
        if (n > 4) {
            // after the tile's counted places, by an atomic; four at a time, since
            // an atomic's answer takes longer than everything else here
            for (int k0 = 0; k0 < n; k0 += 4) {
                long long at[4] = {-1, -1, -1, -1};
                four_tiles(b, k0, n, tilesX, [&](int k, int tile) {
                    at[k] = tileStart[tile] + tileCount[tile] + atomicAdd(&tileFill[tile], 1);
                });
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (at[k] >= 0 && at[k] < capacity) pairs[at[k]] = slot;
            }
        } else if (n > 0) {
            const uint4 q = places[slot];
            const uint32_t in[4] = {q.x, q.y, q.z, q.w};
            long long at[4] = {-1, -1, -1, -1};
            four_tiles(b, 0, n, tilesX, [&](int k, int tile) { at[k] = tileStart[tile] + in[k]; });
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (at[k] >= 0 && at[k] < capacity) pairs[at[k]] = slot;
        }
    };
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
        const uint4 b = boxes[t];
        put(make_uint2(b.x, b.y), 2 * t);
        put(make_uint2(b.z, b.w), 2 * t + 1);
    }
}

// edge (a -> b), counter-clockwise: a centre exactly on it is inside when the
// edge has dy < 0, or dy == 0 and dx > 0
__device__ __forceinline__ bool edge_owns(int ax, int ay, int bx, int by)
{
    const int dx = bx - ax, dy = by - ay;
    return dy < 0 || (dy == 0 && dx > 0);
}

__device__ __forceinline__ long long edge_fn(int ax, int ay, int bx, int by, long long px, long long py)
{
    return (long long)(bx - ax) * (py - ay) - (long long)(by - ay) * (px - ax);
}

// A staged record, prepared by one lane for the tile's 256 pixels:
//  e = edge functions at the tile's first pixel centre, less 1 where a centre on
//      the edge belongs to the other triangle (bit k of `less`), so that inside
//      means e >= 0
//  a, b = their steps per pixel in x and y
//  z = the vertices' depths, area = twice the area in FP32, rarea its reciprocal
// In 32 bits for sub-triangles at most 2^14 sixteenths of a pixel across that
// touch the tile: an edge function within the tile is then below
// 2 (2^14 + 2^9) 2^14 < 2^30, the exact integer the 64-bit form gives.  Others
// (and depths beyond 2) have small = 0 and are evaluated from the record.
struct TileRec {
    int e[3], slot, a[3], less, b[3], small;
    float z[3], area;
    float rarea, pad[3];
};

// Approximate against exact depth (|z| <= 2): below 2^-19.
constexpr float kDepthSlack = 1e-5f;

// One block per tile.  A thread prepares a record, with the warps -- 8 x 4
// pixels each -- that have a pixel it can cover (every edge function non-negative
// at a corner), and each warp goes through its own.  The exact depth (three
// divisions) is formed only where the approximate one is not clearly behind the
// pixel's nearest so far.  1920 x 1080, 331k triangles: 705 us as 16 x 2 pixels a
// warp, every record, 64-bit edge functions; 170 us in this form (70 % of issue
// slots busy).
__global__ void __launch_bounds__(kTile * kTile) k_rs_tiles(const float4 *__restrict__ recs,
                                                            const int *__restrict__ tileCount,
                                                            const int *__restrict__ tileMore,
                                                            const long long *__restrict__ tileStart,
                                                            const int *__restrict__ pairs, int W, int H, int tilesX,
                                                            int clear, const float *__restrict__ mats, float4 *g0,
                                                            float4 *g1, float4 *g2, float4 *g3, float *depth)
{
    __shared__ TileRec s_rec[kChunk];
    __shared__ uint32_t s_warps[kChunk];   // the warps whose pixels a record can touch
    const int tile = blockIdx.x, tx = tile % tilesX, ty = tile / tilesX;
    const int n = tileCount[tile] + tileMore[tile];
    if (n == 0 && !clear) return;
    const long long base = tileStart[tile];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wx = 8 * (warp & 1), wy = 4 * (warp >> 1), lx = wx + (lane & 7), ly = wy + (lane >> 3);
    const int px = tx * kTile + lx, py = ty * kTile + ly;
    const bool inside = px < W && py < H;
    const long long cx = (long long)px * 16 + 8, cy = (long long)py * 16 + 8;
    const int ox = tx * kTile * 16 + 8, oy = ty * kTile * 16 + 8;   // the tile's first centre
    float bz = __int_as_float(0x7f800000);   // +inf
    int bslot = 0x7fffffff;
    for (int c0 = 0; c0 < n; c0 += kChunk) {
        __syncthreads();
        const int m = min(kChunk, n - c0);
        const int sl = threadIdx.x < m ? pairs[base + c0 + threadIdx.x] : -1;
        uint32_t warps = 0;
        if (sl >= 0) {
            const float4 *r = recs + (size_t)kRecF4 * sl;
            const float4 a = __ldg(r), b = __ldg(r + 1), zz = __ldg(r + 2);
            const int X[3] = {__float_as_int(a.x), __float_as_int(a.z), __float_as_int(b.x)};
            const int Y[3] = {__float_as_int(a.y), __float_as_int(a.w), __float_as_int(b.y)};
            const long long area = (long long)(unsigned)__float_as_int(b.z) | ((long long)__float_as_int(b.w) << 32);
            const long long wide = (long long)max(X[0], max(X[1], X[2])) - min(X[0], min(X[1], X[2]));
            const long long high = (long long)max(Y[0], max(Y[1], Y[2])) - min(Y[0], min(Y[1], Y[2]));
            TileRec &q = s_rec[threadIdx.x];
            q.slot = sl;
            q.small = wide <= (1 << 14) && high <= (1 << 14) &&
                      fmaxf(fmaxf(fabsf(zz.x), fabsf(zz.y)), fabsf(zz.z)) <= 2.0f;
            q.less = 0;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int i = (k + 1) % 3, j = (k + 2) % 3;   // edge k runs from vertex i to vertex j
                q.e[k] = q.a[k] = q.b[k] = 0;
                if (q.small) {
                    const int dx = X[j] - X[i], dy = Y[j] - Y[i], less = edge_owns(X[i], Y[i], X[j], Y[j]) ? 0 : 1;
                    q.e[k] = dx * (oy - Y[i]) - dy * (ox - X[i]) - less;
                    q.a[k] = -16 * dy;
                    q.b[k] = 16 * dx;
                    q.less |= less << k;
                }
            }
            q.z[0] = zz.x;
            q.z[1] = zz.y;
            q.z[2] = zz.z;
            q.area = __ll2float_rn(area);
            q.rarea = 1.0f / q.area;
            // the 8 x 4 pixels of warp w: each edge at the corner where it is largest
            int e[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) e[k] = q.e[k] + max(7 * q.a[k], 0) + max(3 * q.b[k], 0);
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                const int x = 8 * (w & 1), y = 4 * (w >> 1);
                int out = 0;
#pragma unroll
                for (int k = 0; k < 3; ++k) out |= e[k] + q.a[k] * x + q.b[k] * y;
                if (out >= 0) warps |= 1u << w;
            }
        }
        s_warps[threadIdx.x] = warps;
        __syncthreads();
        for (int first = 0; first < m; first += 32)
          for (unsigned todo = __ballot_sync(kFullWarp, (s_warps[first + lane] >> warp) & 1u); todo; todo &= todo - 1u) {
            const TileRec &q = s_rec[first + __ffs(todo) - 1];
            float f0, f1, f2;
            if (q.small) {
                const int e0 = q.e[0] + q.a[0] * lx + q.b[0] * ly, e1 = q.e[1] + q.a[1] * lx + q.b[1] * ly,
                          e2 = q.e[2] + q.a[2] * lx + q.b[2] * ly;
                if ((e0 | e1 | e2) < 0 || !inside) continue;
                f0 = __int2float_rn(e0 + (q.less & 1));
                f1 = __int2float_rn(e1 + ((q.less >> 1) & 1));
                f2 = __int2float_rn(e2 + (q.less >> 2));
                if (((f0 * q.z[0] + f1 * q.z[1]) + f2 * q.z[2]) * q.rarea > bz + kDepthSlack) continue;
            } else {
                if (!inside) continue;
                const float4 *r = recs + (size_t)kRecF4 * q.slot;
                const float4 a = __ldg(r), b = __ldg(r + 1);
                const int X0 = __float_as_int(a.x), Y0 = __float_as_int(a.y), X1 = __float_as_int(a.z),
                          Y1 = __float_as_int(a.w), X2 = __float_as_int(b.x), Y2 = __float_as_int(b.y);
                const long long e0 = edge_fn(X1, Y1, X2, Y2, cx, cy), e1 = edge_fn(X2, Y2, X0, Y0, cx, cy),
                                e2 = edge_fn(X0, Y0, X1, Y1, cx, cy);
                if (e0 < 0 || e1 < 0 || e2 < 0) continue;
                if ((e0 == 0 && !edge_owns(X1, Y1, X2, Y2)) || (e1 == 0 && !edge_owns(X2, Y2, X0, Y0)) ||
                    (e2 == 0 && !edge_owns(X0, Y0, X1, Y1)))
                    continue;
                f0 = __ll2float_rn(e0);
                f1 = __ll2float_rn(e1);
                f2 = __ll2float_rn(e2);
            }
            const float l0 = __fdiv_rn(f0, q.area), l1 = __fdiv_rn(f1, q.area), l2 = __fdiv_rn(f2, q.area);
            const float z = __fadd_rn(__fadd_rn(__fmul_rn(l0, q.z[0]), __fmul_rn(l1, q.z[1])), __fmul_rn(l2, q.z[2]));
            if (!(z >= 0.0f && z <= 1.0f)) continue;
            if (z < bz || (z == bz && q.slot < bslot)) {
                bz = z;
                bslot = q.slot;
            }
          }
    }
    if (!inside) return;
    const size_t p = (size_t)py * W + px;
    if (bslot == 0x7fffffff) {
        if (!clear) return;
        const float nan = __int_as_float(0x7fc00000);
        const float4 none = make_float4(nan, nan, nan, nan);
        g0[p] = none;
        g1[p] = none;
        if (g2) g2[p] = none;
        if (g3) g3[p] = none;
        if (depth) depth[p] = 1.0f;
        return;
    }
    if (!clear && !(bz < depth[p])) return;   // GL_LESS against earlier draws
    const float4 *r = recs + (size_t)kRecF4 * bslot;
    const float4 a = r[0], b = r[1], r2 = r[2], r3 = r[3], r4 = r[4], r5 = r[5], r6 = r[6], r7 = r[7], r8 = r[8];
    const int X0 = __float_as_int(a.x), Y0 = __float_as_int(a.y), X1 = __float_as_int(a.z), Y1 = __float_as_int(a.w),
              X2 = __float_as_int(b.x), Y2 = __float_as_int(b.y);
    const long long e0 = edge_fn(X1, Y1, X2, Y2, cx, cy);
    const long long e1 = edge_fn(X2, Y2, X0, Y0, cx, cy);
    const long long e2 = edge_fn(X0, Y0, X1, Y1, cx, cy);
    const long long area = (long long)(unsigned)__float_as_int(b.z) | ((long long)__float_as_int(b.w) << 32);
    const float fa = __ll2float_rn(area);
    const float l0 = __fdiv_rn(__ll2float_rn(e0), fa), l1 = __fdiv_rn(__ll2float_rn(e1), fa),
                l2 = __fdiv_rn(__ll2float_rn(e2), fa);
    const float q0 = __fmul_rn(l0, r2.w), q1 = __fmul_rn(l1, r3.x), q2 = __fmul_rn(l2, r3.y);
    const float d = __fadd_rn(__fadd_rn(q0, q1), q2);
    const float P0[3] = {r4.x, r4.y, r4.z}, P1[3] = {r4.w, r5.x, r5.y}, P2[3] = {r5.z, r5.w, r6.x};
    const float N0[3] = {r6.y, r6.z, r6.w}, N1[3] = {r7.x, r7.y, r7.z}, N2[3] = {r7.w, r8.x, r8.y};
    float P[3], N[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        P[k] = __fdiv_rn(__fadd_rn(__fadd_rn(__fmul_rn(q0, P0[k]), __fmul_rn(q1, P1[k])), __fmul_rn(q2, P2[k])), d);
        N[k] = __fdiv_rn(__fadd_rn(__fadd_rn(__fmul_rn(q0, N0[k]), __fmul_rn(q1, N1[k])), __fmul_rn(q2, N2[k])), d);
    }
    const float *mt = mats + 10 * (size_t)__float_as_int(r3.z);
    if (depth) depth[p] = bz;
    g0[p] = make_float4(P[0], P[1], P[2], mt[6]);
    g1[p] = make_float4(N[0], N[1], N[2], mt[7]);
    if (g2) g2[p] = make_float4(mt[0], mt[1], mt[2], mt[8]);
    if (g3) g3[p] = make_float4(mt[3], mt[4], mt[5], mt[9]);
}

}  // namespace
}  // namespace fdzb

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
static_assert(sizeof(fdzb_raster_desc) == 240, "fdzb_raster_desc layout");
static_assert(sizeof(fdzb_raster_stats) == 64, "fdzb_raster_stats layout");

struct fdzb_raster {
    int device = 0, sms = 148;
    cudaStream_t own = nullptr, stream = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr, counted = nullptr;
    // records, places and boxes of slotCap slots, one allocation (a cudaMalloc beyond
    // the small ones takes 0.36 ms, whatever its size)
    char *slots = nullptr;
    size_t slotCap = 0;
    // counters, then tileCount, tileMore, tileFill (cleared with them) and tileStart
    char *tiles = nullptr;
    size_t tileCap = 0;
    int *pairs = nullptr;
    size_t pairCap = 0;
    fdzb::RasterCounters *hCtr = nullptr;
    fdzb_raster_stats stats{};
    bool pending = false;
};

namespace {

int rfail(int code, const std::string &msg) { return fdzb::set_error(code, "fdzb_raster: " + msg); }

#define RS_CUDA(call)                                                                         \
    do {                                                                                      \
        cudaError_t _e = (call);                                                              \
        if (_e != cudaSuccess) return rfail(FDZB_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
    } while (0)

int grow(void **p, size_t &cap, size_t need, size_t elem)
{
    if (need <= cap) return FDZB_OK;
    if (*p) cudaFree(*p);
    *p = nullptr;
    cap = 0;
    // a quarter to spare, or what the draw needs where that is all there is
    size_t n = need + need / 4 + 64;
    if (cudaMalloc(p, n * elem) != cudaSuccess) {
        cudaGetLastError();
        n = need;
        if (cudaMalloc(p, n * elem) != cudaSuccess) {
            *p = nullptr;
            cudaGetLastError();
            return rfail(FDZB_ERR_NO_MEMORY, "device allocation failed");
        }
    }
    cap = n;
    return FDZB_OK;
}

constexpr size_t kCtrBytes = 256;
static_assert(sizeof(fdzb::RasterCounters) <= kCtrBytes, "counters' place before the tile arrays");

int finish(fdzb_raster *r)
{
    if (!r->pending) return FDZB_OK;
    RS_CUDA(cudaEventSynchronize(r->e1));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, r->e0, r->e1);
    r->stats.ms = ms;
    r->pending = false;
    return FDZB_OK;
}

}  // namespace

extern "C" {

int fdzb_raster_create(fdzb_raster **out, int device)
{
    if (!out) return rfail(FDZB_ERR_INVALID_ARG, "out is NULL");
    *out = nullptr;
    int dev = device;
    if (dev < 0) RS_CUDA(cudaGetDevice(&dev));
    RS_CUDA(cudaSetDevice(dev));
    fdzb_raster *r = new fdzb_raster();
    r->device = dev;
    if (cudaStreamCreateWithFlags(&r->own, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&r->e0) != cudaSuccess || cudaEventCreate(&r->e1) != cudaSuccess ||
        cudaEventCreateWithFlags(&r->counted, cudaEventDisableTiming) != cudaSuccess ||
        cudaMallocHost(&r->hCtr, sizeof(fdzb::RasterCounters)) != cudaSuccess) {
        cudaGetLastError();
        fdzb_raster_destroy(r);
        return rfail(FDZB_ERR_CUDA, "could not create the rasteriser's stream, events or buffers");
    }
    cudaDeviceGetAttribute(&r->sms, cudaDevAttrMultiProcessorCount, dev);
    r->stream = r->own;
    *out = r;
    return FDZB_OK;
}

int fdzb_raster_destroy(fdzb_raster *r)
{
    if (!r) return FDZB_OK;
    cudaSetDevice(r->device);
    if (r->stream) cudaStreamSynchronize(r->stream);
    cudaFree(r->slots);
    cudaFree(r->tiles);
    cudaFree(r->pairs);
    if (r->hCtr) cudaFreeHost(r->hCtr);
    if (r->e0) cudaEventDestroy(r->e0);
    if (r->e1) cudaEventDestroy(r->e1);
    if (r->counted) cudaEventDestroy(r->counted);
    if (r->own) cudaStreamDestroy(r->own);
    delete r;
    return FDZB_OK;
}

int fdzb_raster_set_stream(fdzb_raster *r, void *stream)
{
    if (!r) return rfail(FDZB_ERR_INVALID_ARG, "handle is NULL");
    if (int rc = finish(r)) return rc;
    r->stream = stream ? (cudaStream_t)stream : r->own;
    return FDZB_OK;
}

int fdzb_raster_sync(fdzb_raster *r)
{
    if (!r) return rfail(FDZB_ERR_INVALID_ARG, "handle is NULL");
    cudaSetDevice(r->device);
    return finish(r);
}

int fdzb_raster_get_stats(fdzb_raster *r, fdzb_raster_stats *st)
{
    if (!r || !st) return rfail(FDZB_ERR_INVALID_ARG, "NULL argument");
    if (int rc = fdzb_raster_sync(r)) return rc;
    *st = r->stats;
    return FDZB_OK;
}

int fdzb_raster_draw(fdzb_raster *r, const fdzb_raster_desc *d)
{
    using namespace fdzb;
    if (!r || !d) return rfail(FDZB_ERR_INVALID_ARG, "NULL argument");
    if (d->W < 1 || d->H < 1 || d->W > 16384 || d->H > 16384) return rfail(FDZB_ERR_INVALID_ARG, "W, H must be in 1..16384");
    if (d->n_tri < 0 || d->n_vtx < 0) return rfail(FDZB_ERR_INVALID_ARG, "negative count");
    if (d->n_tri > (1 << 29)) return rfail(FDZB_ERR_INVALID_ARG, "too many triangles (max 2^29)");
    if (d->n_tri > 0 && (!d->d_vtx || !d->d_idx)) return rfail(FDZB_ERR_INVALID_ARG, "NULL vertex or index buffer");
    if (d->vtx_stride_bytes < 12 || d->vtx_stride_bytes % 4) return rfail(FDZB_ERR_INVALID_ARG, "vertex stride must be >= 12, a multiple of 4");
    const int strideF = d->vtx_stride_bytes / 4;
    if (d->pos_offset < 0 || d->nrm_offset < 0 || d->pos_offset + 3 > strideF || d->nrm_offset + 3 > strideF)
        return rfail(FDZB_ERR_INVALID_ARG, "position / normal offsets outside the vertex");
    if (!d->d_materials || d->n_materials < 1) return rfail(FDZB_ERR_INVALID_ARG, "at least one material is required");
    if (!d->d_g0 || !d->d_g1) return rfail(FDZB_ERR_INVALID_ARG, "g0 and g1 are required");
    for (const void *p : {(const void *)d->d_g0, (const void *)d->d_g1, (const void *)d->d_g2, (const void *)d->d_g3})
        if ((uintptr_t)p & 15) return rfail(FDZB_ERR_INVALID_ARG, "G-buffer targets must be 16-byte aligned float4 arrays");
    if (!d->clear && !d->d_depth) return rfail(FDZB_ERR_INVALID_ARG, "drawing without clear needs the earlier draw's depth buffer");
    cudaSetDevice(r->device);
    if (int rc = finish(r)) return rc;
    cudaStreamCaptureStatus capture;
    RS_CUDA(cudaStreamIsCapturing(r->stream, &capture));
    if (capture != cudaStreamCaptureStatusNone)
        return rfail(FDZB_ERR_CUDA, "a draw waits for its tile-list size and cannot be captured");

    const int W = d->W, H = d->H;
    const size_t S = (size_t)W * H;
    const int tilesX = (W + 15) / 16, tilesY = (H + 15) / 16;
    const size_t nTiles = (size_t)tilesX * tilesY;
    const size_t T = (size_t)d->n_tri;
    constexpr size_t kRecBytes = kRecF4 * sizeof(float4), kSlotBytes = kRecBytes + sizeof(uint4) + sizeof(uint2);
    if (int rc = grow((void **)&r->slots, r->slotCap, 2 * std::max<size_t>(T, 1), kSlotBytes)) return rc;
    float4 *recs = (float4 *)r->slots;
    uint4 *places = (uint4 *)(r->slots + kRecBytes * r->slotCap);
    uint2 *boxes = (uint2 *)(r->slots + (kRecBytes + sizeof(uint4)) * r->slotCap);
    // the four arrays of a capacity of r->tileCap tiles
    if (nTiles > r->tileCap) {
        size_t bytes = 0;
        const size_t cap = (nTiles + nTiles / 4 + 64) / 2 * 2;
        cudaFree(r->tiles);
        r->tiles = nullptr;
        r->tileCap = 0;
        if (int rc = grow((void **)&r->tiles, bytes, kCtrBytes + cap * 20 + 8, 1)) return rc;
        r->tileCap = cap;
    }
    RasterCounters *ctr = (RasterCounters *)r->tiles;
    int *tileCount = (int *)(r->tiles + kCtrBytes), *tileMore = tileCount + nTiles, *tileFill = tileMore + nTiles;
    const size_t cleared = kCtrBytes + (12 * nTiles + 7) / 8 * 8;
    long long *tileStart = (long long *)(r->tiles + cleared);
    cudaStream_t s = r->stream;
    const int sm = r->sms;
    RasterMats mats;
    std::memcpy(mats.model, d->model, sizeof(mats.model));
    std::memcpy(mats.viewProj, d->view_proj, sizeof(mats.viewProj));
    RS_CUDA(cudaEventRecord(r->e0, s));
    RS_CUDA(cudaMemsetAsync(r->tiles, 0, cleared, s));
    if (T > 0) {
        const int g = (int)std::min<long long>((d->n_tri + 127) / 128, (long long)sm * 16);
        const bool wide = strideF == 8 && d->pos_offset == 0 && d->nrm_offset == 5 && !((uintptr_t)d->d_vtx & 15);
        auto setup = wide ? k_rs_setup<1> : k_rs_setup<0>;
        setup<<<g, 128, 0, s>>>(d->d_vtx, d->n_vtx, strideF, d->pos_offset, d->nrm_offset, d->d_idx, d->n_tri,
                                d->d_tri_material, d->n_materials, mats, W, H, tilesX, recs, boxes, places, tileCount,
                                tileMore, ctr);
    }
    RS_CUDA(cudaGetLastError());
    // The lists' length sizes their buffer, and a draw of more than 2^31 pairs is
    // refused before anything is drawn: the host waits for the counters.  A buffer
    // sized by guess saved nothing (34k triangles: 93 us a draw, 92 with the wait)
    // and cost draws that outgrew it: 34 ms instead of 2.3 where a view of 100k
    // triangles moved up to them.
    *r->hCtr = RasterCounters{};
    if (T > 0) {
        k_rs_lists<<<(unsigned)((nTiles + 255) / 256), 256, 0, s>>>(tileCount, tileMore, tileStart, (int)nTiles, ctr, r->hCtr);
        RS_CUDA(cudaGetLastError());
        RS_CUDA(cudaEventRecord(r->counted, s));
        RS_CUDA(cudaEventSynchronize(r->counted));
    }
    const RasterCounters c = *r->hCtr;
    r->stats = fdzb_raster_stats{};
    r->stats.triangles = d->n_tri;
    r->stats.sub_triangles = (int64_t)c.subTris;
    r->stats.dropped = (int64_t)c.dropped;
    r->stats.tile_pairs = (int64_t)c.pairs;
    r->stats.bad_indices = (int64_t)c.badIdx;
    r->stats.bad_materials = (int64_t)c.badMat;
    r->stats.tiles_x = tilesX;
    r->stats.tiles_y = tilesY;
    if (c.pairs > 0x7fffffffull) return rfail(FDZB_ERR_CAPACITY, "more than 2^31 tile pairs in one draw");
    if (c.pairs > 0) {
        if (int rc = grow((void **)&r->pairs, r->pairCap, (size_t)c.pairs, sizeof(int))) return rc;
        k_rs_scatter<<<(int)std::min<long long>((d->n_tri + 255) / 256, (long long)sm * 8), 256, 0, s>>>(
            (const uint4 *)boxes, places, d->n_tri, tilesX, tileCount, tileStart, tileFill, r->pairs, (long long)r->pairCap);
        k_rs_tiles<<<(unsigned)nTiles, 256, 0, s>>>(recs, tileCount, tileMore, tileStart, r->pairs, W, H, tilesX, d->clear,
                                                    d->d_materials, (float4 *)d->d_g0, (float4 *)d->d_g1,
                                                    (float4 *)d->d_g2, (float4 *)d->d_g3, d->d_depth);
    } else if (d->clear) {
        const int g = (int)std::min<size_t>((S + 255) / 256, (size_t)sm * 8);
        k_rs_clear<<<g, 256, 0, s>>>((int)S, (float4 *)d->d_g0, (float4 *)d->d_g1, (float4 *)d->d_g2,
                                     (float4 *)d->d_g3, d->d_depth);
    }
    RS_CUDA(cudaGetLastError());
    RS_CUDA(cudaEventRecord(r->e1, s));
    r->pending = true;
    return FDZB_OK;
}

}  // extern "C"
