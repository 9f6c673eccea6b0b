// fdzb_occlusion.cuh -- the exact pair tests and what the occlusion kernels
// share (stages c + d).
//
// Reference: shadowCal_per_sample_kernel (K/Step5_2_shadowCalPerSample.inl:37-231),
// one thread per sample walking its bin's triangle list through texture fetches.
//
// Here a warp owns a work item: samples of one bin, 32 at a time, a lane each;
// the bin's triangles are staged into shared memory kOccChunk at a time and
// every lane tests its own sample against them, until its light rows are all
// full (the reference's early-out) or the list ends.  The mask is the OR over
// the tested triangles, so it is independent of their order.  The edge-mask
// kernel is in fdzb_edge_masks.cuh; this file has the reference's pair test
// itself (pair_test), the ray-cast cross-check and the lane-per-pair schedule.
#pragma once
#include "fdzb_device.cuh"

namespace fdzb {

#ifndef FDZB_OCC_MINBLOCKS
#define FDZB_OCC_MINBLOCKS 7
#endif

#ifndef FDZB_OCC_ITEM
#define FDZB_OCC_ITEM 32
#endif
#ifndef FDZB_OCC_CHUNK
#define FDZB_OCC_CHUNK 32
#endif


constexpr int kOccWarps = 4;
constexpr int kOccThreads = kOccWarps * 32;
constexpr int kOccChunk = FDZB_OCC_CHUNK;
static_assert(kOccChunk >= 1 && kOccChunk <= 32, "a chunk is staged one triangle per lane");
constexpr int kItemSamples = FDZB_OCC_ITEM;

// Row words: uint32_t (grids up to 32 x 32, the reference's U32) or
// unsigned long long (up to 64 x 64, the reference's template at T = U64).
template <class R> struct RowWord;
template <> struct RowWord<uint32_t> {
    static constexpr int kBits = 32;
    static constexpr int kWarps = 4;
    static constexpr int kMinBlocks = FDZB_OCC_MINBLOCKS;
    __device__ static int lowest(uint32_t v) { return __ffs(v) - 1; }
    __device__ static int popc(uint32_t v) { return __popc(v); }
    __device__ static uint32_t fullCols(const LightParams &L) { return L.full; }
    __device__ static uint32_t fullRows(const LightParams &L) { return (uint32_t)L.fullRows; }
};
template <> struct RowWord<unsigned long long> {
    static constexpr int kBits = 64;
    // 16 KB of rows a warp: 11 blocks of one warp fill an SM's shared memory, 5 of
    // two leave room (64 x 48 light, 1920 x 1080: 19.5 -> 18.5 ms)
    static constexpr int kWarps = 1;
    static constexpr int kMinBlocks = 11;
    __device__ static int lowest(unsigned long long v) { return __ffsll((long long)v) - 1; }
    __device__ static int popc(unsigned long long v) { return __popcll(v); }
    __device__ static unsigned long long fullCols(const LightParams &L) { return L.fullCols; }
    __device__ static unsigned long long fullRows(const LightParams &L) { return L.fullRows; }
};
typedef unsigned long long u64;

// K/Step5_2_shadowCalPerSample.inl:14-33: the places i in [0, count) where
// D + slope i >= 0, from the signs at both ends and the round-up conversion of
// q = -D / slope (the same integer as the reference's truncating conversion of
// ceilf(q)); PTX shl: amounts >= the word width give 0.  npart counts the
// partial masks (COUNT).
template <class R, int COUNT>
__device__ __forceinline__ R row_mask(float D, float slopeNm1, float slope, R full, uint32_t &npart)
{
    const bool f1 = D >= 0.0f;
    const bool f2 = __fadd_rn(slopeNm1, D) >= 0.0f;
    if (f1 && f2) return full;
    if (!f1 && !f2) return R(0);
    if (COUNT) ++npart;
    const float q = __fdiv_rn(-D, slope);
    const int k = __float2int_ru(q);
    R m = ((unsigned)k >= (unsigned)RowWord<R>::kBits) ? R(0) : (R(1) << k);
    m -= R(1);
    if (!f1) m = ~m;
    return m & full;
}

// K/Step5_2_shadowCal.inl:213-222
__device__ __forceinline__ bool point_in_tri(f3 A, f3 B, f3 C, f3 P)
{
    const f3 N1 = cross3(sub3(B, A), sub3(P, B));
    const f3 N2 = cross3(sub3(C, B), sub3(P, C));
    if (dot3(N1, N2) < 0.0f) return false;
    const f3 N3 = cross3(sub3(A, C), sub3(P, A));
    if (dot3(N2, N3) < 0.0f) return false;
    return true;
}

// Staged triangle, 7 x float4:
//  p0 = (aabb min x, min y, max x, max y)   p1 = (minz, v0)
//  p2 = (v1, v2.x)   p3 = (v2.y, v2.z, n.x, n.y)   p4 = (n.z, e01)
//  p5 = (e12, e20.x) p6 = (e20.y, e20.z, maxz, 0)
struct StagedTri {
    float4 p[7];
};

__device__ __forceinline__ void stage_triangle(StagedTri &dst, const float4 *__restrict__ rec, int tri)
{
    const float4 q0 = __ldg(rec + 4 * (size_t)tri);
    const float4 q1 = __ldg(rec + 4 * (size_t)tri + 1);
    const float4 q2 = __ldg(rec + 4 * (size_t)tri + 2);
    const float4 q3 = __ldg(rec + 4 * (size_t)tri + 3);
    const f3 v0 = mk3(q0.x, q0.y, q0.z), v1 = mk3(q1.x, q1.y, q1.z), v2 = mk3(q2.x, q2.y, q2.z);
    const f3 n = cross3(sub3(v1, v0), sub3(v2, v1));   // K/Step5_2_shadowCalPerSample.inl:130
    const f3 e01 = sub3(v0, v1), e12 = sub3(v1, v2), e20 = sub3(v2, v0);  // a - b of :7
    dst.p[0] = q3;
    dst.p[1] = make_float4(q0.w, v0.x, v0.y, v0.z);
    dst.p[2] = make_float4(v1.x, v1.y, v1.z, v2.x);
    dst.p[3] = make_float4(v2.y, v2.z, n.x, n.y);
    dst.p[4] = make_float4(n.z, e01.x, e01.y, e01.z);
    dst.p[5] = make_float4(e12.x, e12.y, e12.z, e20.x);
    dst.p[6] = make_float4(e20.y, e20.z, q1.w, 0.0f);
}

struct LaneSample {
    f3 Q, L0Q;
    float spx, spy, spz, spw, spZ;
};

__device__ __forceinline__ void load_sample(LaneSample &s, const FrameDesc &fr, const FrameState &st,
                                            int local)
{
    const float4 P = __ldg(fr.pos + local);
    s.Q = mk3(P.x, P.y, P.z);
    const f3 r = light_project(fr.light.mat, s.Q);
    s.spx = r.x;
    s.spy = r.y;
    s.spz = __fsub_rn(__fadd_rn(r.x, __fdiv_rn(fr.light.RF[0], r.z)), st.subx);
    s.spw = __fsub_rn(__fadd_rn(r.y, __fdiv_rn(fr.light.RF[1], r.z)), st.suby);
    s.spZ = r.z;
    s.L0Q = sub3(ld3(fr.light.ur), s.Q);
}

// Light grid constants of a frame, in the form the pair tests use them.
template <class R> struct GridC {
    int NR, NC;             // rows (along x_delt), columns (along y_delt)
    float nrm1, ncm1;       // NR - 1, NC - 1
    R FR, FC;               // NR and NC low bits
};
template <class R> __device__ __forceinline__ GridC<R> grid_of(const FrameDesc &fr)
{
    GridC<R> g;
    g.NR = fr.light.N;
    g.NC = fr.light.NC;
    g.nrm1 = (float)(g.NR - 1);
    g.ncm1 = (float)(g.NC - 1);
    g.FR = RowWord<R>::fullRows(fr.light);
    g.FC = RowWord<R>::fullCols(fr.light);
    return g;
}

// One sample/triangle pair (K/Step5_2_shadowCalPerSample.inl:120-222).  Rows r
// step along x_delt (A), columns c along y_delt (B); the row filter bounds the
// column term with B*(NC-1) and the rows with A*(NR-1), which for the
// reference's square grids are its own expressions.  With the depth plane, a
// fourth plane -n.(L - v0), oriented like the edges, keeps light samples on
// the sample's side of the triangle unoccluded (the test of the reference's
// per-bin kernel, K/Step5_2_shadowCal.inl:667-674, 838) for triangles that
// reach the light plane (min depth <= 0: occluders behind the light) or the
// sample's depth (the per-bin kernel's own condition); a triangle strictly
// between them needs no such test.  `open`: the light rows wanted (others are left
// as they are).  The caller has found that the pair passes the pre-cull.
template <class R, int DEPTH, int COUNT>
__device__ __forceinline__ void pair_test(const StagedTri &T, const LaneSample &s, f3 xd, f3 yd, f3 ur,
                                          float esp, const GridC<R> &g, R (*rows)[32], int lane, R open,
                                          R &fullRows, uint32_t &nrows, uint32_t &npart)
{
    const float4 p1 = T.p[1];
    const float4 p2 = T.p[2], p3 = T.p[3], p4 = T.p[4], p5 = T.p[5], p6 = T.p[6];
    const f3 v0 = mk3(p1.y, p1.z, p1.w), v1 = mk3(p2.x, p2.y, p2.z), v2 = mk3(p2.w, p3.x, p3.y);
    const f3 n = mk3(p3.z, p3.w, p4.x);
    const f3 e01 = mk3(p4.y, p4.z, p4.w), e12 = mk3(p5.x, p5.y, p5.z), e20 = mk3(p5.w, p6.x, p6.y);
    const f3 Q = s.Q;
    const float dir = dot3(sub3(Q, v0), n);
    if (fabsf(dir) < esp && point_in_tri(v0, v1, v2, Q)) return;
    // orientation: the reference negates t0, t1 and L0 - Q when dir < 0
    const bool neg = dir < 0.0f;
    const f3 t0 = neg ? mk3(-xd.x, -xd.y, -xd.z) : xd;
    const f3 t1 = neg ? mk3(-yd.x, -yd.y, -yd.z) : yd;
    const f3 lq = neg ? mk3(-s.L0Q.x, -s.L0Q.y, -s.L0Q.z) : s.L0Q;
    // getPlaneDiscriminant for (v0,v1), (v1,v2), (v2,v0): n_k = cross(b - Q, a - b)
    float A[4], B[4], C[4];
    const f3 to[3] = {sub3(v1, Q), sub3(v2, Q), sub3(v0, Q)}, along[3] = {e01, e12, e20};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const f3 nk = cross3(to[k], along[k]);
        A[k] = dot3(nk, t0);
        B[k] = dot3(nk, t1);
        C[k] = dot3(nk, lq);
    }
    const bool dp = DEPTH && (p1.x <= 0.0f || p6.z >= s.spZ);
    if (dp) {
        const f3 m = mk3(-n.x, -n.y, -n.z);
        const f3 lv0 = sub3(ur, v0);
        const f3 lv = neg ? mk3(-lv0.x, -lv0.y, -lv0.z) : lv0;
        A[3] = dot3(m, t0);
        B[3] = dot3(m, t1);
        C[3] = dot3(m, lv);
    }
    // row filter (:176-191).  IEEE divisions throughout: this test is the fast
    // one's fallback, and its size in the instruction cache matters more than its
    // speed (hoisted reciprocals in a second row loop: view of 331k triangles 1.41
    // ms occlusion, against 1.31 ms without them).
    R vr = open & ~fullRows;
#pragma unroll
    for (int k = 0; k < 3 + DEPTH; ++k)
        if (k < 3 || dp) vr &= row_mask<R, COUNT>(__fadd_rn(B[k] > 0.0f ? __fmul_rn(B[k], g.ncm1) : 0.0f, C[k]), __fmul_rn(A[k], g.nrm1),
                                 A[k], g.FR, npart);
    // rows (:204-222)
    while (vr) {
        const int r = RowWord<R>::lowest(vr);
        vr &= vr - R(1);
        if (COUNT) ++nrows;
        const float fr = (float)r;
        R m = g.FC;
#pragma unroll
        for (int k = 0; k < 3 + DEPTH; ++k)
            if (k < 3 || dp) m &= row_mask<R, COUNT>(__fadd_rn(__fmul_rn(A[k], fr), C[k]), __fmul_rn(B[k], g.ncm1), B[k], g.FC, npart);
        const R nv = rows[r][lane] | m;
        rows[r][lane] = nv;
        if (nv == g.FC) fullRows |= R(1) << r;
    }
}

// Ray-cast pair test: the reference's REF_CAL cross-check (refCal_kernel and
// intersect_triangle_branchless, K/Step5_2_calRef.inl:1-126).  For every light
// sample not yet occluded, a ray from the sample's position to the light
// sample's position; occluded when it meets the triangle with 1e-3 < t < dist.
// The reference numbers light sample (i along the light's height, j along its
// width) as i*W + j and places it at upRight + x_delt*j + y_delt*i
// (FS/api.cpp:351-357); here it is stored in this library's mask layout, row
// r = j (width), column c = i (height), so that the ray-cast and edge-function
// masks compare bit for bit.  Same pre-cull as the reference's checker: the
// sample's rectangle inside the triangle's AABB and minz - 1e-3 (in double, as
// the reference's double literal makes it) not above the sample's depth.
template <class R, int COUNT>
__device__ __forceinline__ int raycast_pair(const StagedTri &T, const LaneSample &s, f3 ur, f3 xd, f3 yd,
                                            const GridC<R> &g, R (*rows)[32], int lane, R &fullRows,
                                            uint32_t &nrows)
{
    const float4 p0a = T.p[0];
    const float4 p1a = T.p[1];
    if (!(s.spz <= p0a.z && s.spw <= p0a.w && s.spx >= p0a.x && s.spy >= p0a.y)) return 0;
    if ((double)p1a.x - 1e-3 > (double)s.spZ) return 0;
    const float4 p2a = T.p[2], p3a = T.p[3];
    const f3 v0 = mk3(p1a.y, p1a.z, p1a.w), v1 = mk3(p2a.x, p2a.y, p2a.z), v2 = mk3(p2a.w, p3a.x, p3a.y);
    const f3 e0 = sub3(v1, v0);
    const f3 e1 = sub3(v0, v2);
    const f3 n = cross3(e1, e0);
    const f3 q0 = sub3(v0, s.Q);
    const float tmin = 1e-3f;
    for (int r = 0; r < g.NR; ++r) {
        const R have = rows[r][lane];
        if (have == g.FC) continue;
        if (COUNT) ++nrows;
        const f3 lr = add3(ur, mul3(xd, (float)r));   // upRight + x_delt * j
        R add = 0;
        for (int c = 0; c < g.NC; ++c) {
            if (have & (R(1) << c)) continue;
            const f3 lp = add3(lr, mul3(yd, (float)c));   // ... + y_delt * i
            const f3 L = sub3(lp, s.Q);
            const float dist = __fsqrt_rn(dot3(L, L));
            const f3 dir = mk3(__fdiv_rn(L.x, dist), __fdiv_rn(L.y, dist), __fdiv_rn(L.z, dist));
            const float inv = __fdiv_rn(1.0f, dot3(n, dir));
            const f3 e2 = mul3(q0, inv);
            const f3 iv = cross3(dir, e2);
            const float beta = dot3(iv, e1);
            const float gamma = dot3(iv, e0);
            const float t = dot3(n, e2);
            if ((t < dist) & (t > tmin) & (beta >= 0.0f) & (gamma >= 0.0f) & (__fadd_rn(beta, gamma) <= 1.0f))
                add |= R(1) << c;
        }
        if (add) {
            const R nv = have | add;
            rows[r][lane] = nv;
            if (nv == g.FC) fullRows |= R(1) << r;
        }
    }
    return 1;
}

// Bits [pos, pos + n) of a packed mask (n <= 64), LSB first.
__device__ __forceinline__ u64 mask_bits(const uint32_t *w, int pos, int n)
{
    u64 v = 0;
    int got = 0;
    while (got < n) {
        const int wi = (pos + got) >> 5, o = (pos + got) & 31;
        const int take = min(32 - o, n - got);
        const uint32_t part = (w[wi] >> o) & (take == 32 ? 0xffffffffu : ((1u << take) - 1u));
        v |= (u64)part << got;
        got += take;
    }
    return v;
}

// Shadow = set bits / (rows * cols) (:226-231) and the packed mask, bit r * NC + c.
template <class R>
__device__ __forceinline__ void write_result(const FrameDesc &fr, int local, const GridC<R> &g, R (*rows)[32],
                                             int lane)
{
    int cnt = 0;
    for (int r = 0; r < g.NR; ++r) cnt += RowWord<R>::popc(rows[r][lane]);
    fr.shadow[local] = __fdiv_rn((float)cnt, (float)(g.NR * g.NC));   // :226-231
    if (fr.masks) {
        uint32_t *mo = fr.masks + (size_t)local * fr.maskWords;
        u64 acc = 0;
        int bit = 0, wi = 0;
        for (int r = 0; r < g.NR; ++r) {
            u64 v = (u64)rows[r][lane];
            int rem = g.NC;
            while (rem > 0) {
                const int take = min(rem, 32);
                const u64 part = v & (take == 32 ? 0xffffffffull : ((1ull << take) - 1ull));
                acc |= part << bit;
                bit += take;
                if (bit >= 32) {
                    mo[wi++] = (uint32_t)acc;
                    acc >>= 32;
                    bit -= 32;
                }
                v >>= take;
                rem -= take;
            }
        }
        if (bit > 0) mo[wi] = (uint32_t)acc;
    }
}

// Rows of a sample from its packed mask (bit r*NC + c is row r, column c), for
// a launch that accumulates into masks of an earlier triangle pass.  Returns
// the set of full rows.
template <class R>
__device__ __forceinline__ R load_rows(const FrameDesc &fr, int local, const GridC<R> &g, R (*rows)[32], int lane)
{
    const uint32_t *mi = fr.masks + (size_t)local * fr.maskWords;
    R fullRows = 0;
    for (int r = 0; r < g.NR; ++r) {
        const R v = (R)mask_bits(mi, r * g.NC, g.NC) & g.FC;
        rows[r][lane] = v;
        if (v == g.FC) fullRows |= R(1) << r;
    }
    return fullRows;
}

// First contact of a sample with the pipeline's occlusion stage: rows cleared,
// or loaded from the masks of an earlier triangle pass.
template <class R>
__device__ __forceinline__ R init_rows(const FrameDesc &fr, int local, const GridC<R> &g, R (*rows)[32], int lane)
{
    if (fr.accumulate) return load_rows<R>(fr, local, g, rows, lane);
    for (int r = 0; r < g.NR; ++r) rows[r][lane] = 0;
    return 0;
}

__device__ __forceinline__ void write_zero(const FrameDesc &fr, int local)
{
    fr.shadow[local] = 0.0f;
    if (fr.masks) {
        uint32_t *mo = fr.masks + (size_t)local * fr.maskWords;
        for (int w = 0; w < fr.maskWords; ++w) mo[w] = 0u;
    }
}

// Samples per work item of a frame (FrameDesc::occItem; 32 if out of range).
__device__ __forceinline__ int item_samples(const FrameDesc &fr)
{
    const int v = fr.occItem;
    return (v == 64 || v == 128) ? v : kItemSamples;
}

// Triangles staged per chunk of a frame (FrameDesc::occChunk, within [1, kOccChunk]).
__device__ __forceinline__ int chunk_of(const FrameDesc &fr)
{
    const int v = fr.occChunk;
    return (v >= 1 && v <= kOccChunk) ? v : kOccChunk;
}

// k_items: one thread per bin; a bin with n samples yields ceil(n / item) items
// (bin, first sample offset, frame, triangle count), item = the frame's samples
// per work item.
__global__ void k_items(const FrameDesc *__restrict__ frames, int32_t *__restrict__ bss,
                        int32_t *__restrict__ bse, int32_t *__restrict__ bts,
                        int32_t *__restrict__ bte, const int *__restrict__ binBases, int nframes,
                        int totalBins, int4 *__restrict__ items, int capacity, Counters *ctr)
{
    const int lane = threadIdx.x & 31;
    // segments no element reached hold (kSegAbsent, 0): (0, 0), as the
    // reference's pre-zeroed arrays (the samples' array has the extra slot of
    // the unbinned samples)
    if (blockIdx.x == 0 && threadIdx.x == 0 && bss[totalBins] == kSegAbsent) bss[totalBins] = bse[totalBins] = 0;
    for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < totalBins;
         base += gridDim.x * blockDim.x) {
        const int b = base + lane;
        int n = 0, f = 0, isz = kItemSamples;
        if (b < totalBins) {
            if (bss[b] == kSegAbsent) bss[b] = bse[b] = 0;
            if (bts[b] == kSegAbsent) bts[b] = bte[b] = 0;
            const int cnt = bse[b] - bss[b];
            if (cnt > 0) {
                f = frame_of(binBases, nframes, b);
                isz = item_samples(frames[f]);
                n = (cnt + isz - 1) / isz;
            }
        }
        int x = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFullWarp, x, o);
            if (lane >= o) x += y;
        }
        const int tot = __shfl_sync(kFullWarp, x, 31);
        int wbase = 0;
        if (lane == 0 && tot) wbase = atomicAdd(&ctr->itemCount, tot);
        wbase = __shfl_sync(kFullWarp, wbase, 0);
        if (n) {
            const int nt = bte[b] - bts[b];
            for (int k = 0; k < n; ++k) {
                const int slot = wbase + x - n + k;
                if (slot < capacity) items[slot] = make_int4(b, isz * k, f, nt);
            }
        }
    }
}

// A warp's work item: samples [sLo, sHi) of the sorted list, all of one bin,
// against the bin's triangles [tS, tS + nT).
struct OccItem {
    int frame, sLo, sHi, tS, nT;
};

// Takes the next item with triangles from the work queue (lane 0's ticket);
// items of bins without triangles get their zero shadows here.  False at the
// queue's end.  TEAM: the block's warps take one item together (thread 0's
// ticket; every warp enters and leaves with the others).
template <int TEAM = 0>
__device__ __forceinline__ bool next_item(OccItem &w, const FrameDesc *__restrict__ frames,
                                          const int4 *__restrict__ items, int itemCapacity, Counters *ctr,
                                          const int32_t *__restrict__ bss, const int32_t *__restrict__ bse,
                                          const int32_t *__restrict__ bts, const int32_t *__restrict__ bte,
                                          int totalBins, int nframes, const uint32_t *__restrict__ sortedVals,
                                          int lane)
{
    const int nitems = min(*(volatile const int *)&ctr->itemCount, itemCapacity);
    for (;;) {
        int it = 0;
        if constexpr (TEAM) {
            __shared__ int s_item;
            __syncthreads();
            if (threadIdx.x == 0) s_item = atomicAdd(&ctr->itemCursor, 1);
            __syncthreads();
            it = s_item;
        } else {
            if (lane == 0) it = atomicAdd(&ctr->itemCursor, 1);
            it = __shfl_sync(kFullWarp, it, 0);
        }
        if (it >= nitems) return false;
        const int4 item = items[it];
        const int bin = item.x;
        w.frame = item.z;
        if ((unsigned)bin >= (unsigned)totalBins || (unsigned)w.frame >= (unsigned)nframes) {
            if (lane == 0) atomicOr(&ctr->errorFlags, (int)ERR_INTERNAL);
            continue;
        }
        const FrameDesc &fr = frames[w.frame];
        w.sLo = bss[bin] + item.y;
        w.sHi = min(w.sLo + item_samples(fr), bse[bin]);
        w.tS = bts[bin];
        w.nT = bte[bin] - w.tS;
        if (w.nT > 0) return true;
        // no triangle in this bin: shadow 0 -- or, in a later triangle pass,
        // the result of the earlier passes, left as it is
        if (!fr.accumulate && (!TEAM || threadIdx.x < 32)) {
            for (int k = w.sLo + lane; k < w.sHi; k += 32) {
                const int local = (int)sortedVals[k] - fr.sampleBase;
                if ((unsigned)local < (unsigned)(fr.W * fr.H)) write_zero(fr, local);
                else atomicOr(&ctr->errorFlags, (int)ERR_INTERNAL);
            }
        }
    }
}

// The frame's sample at place k of the sorted list; false past the item's end.
__device__ __forceinline__ bool item_sample(int &local, const uint32_t *__restrict__ sortedVals, int k, int sHi,
                                            const FrameDesc &fr, Counters *ctr)
{
    if (k >= sHi) return false;
    local = (int)sortedVals[k] - fr.sampleBase;
    if ((unsigned)local < (unsigned)(fr.W * fr.H)) return true;
    atomicOr(&ctr->errorFlags, (int)ERR_INTERNAL);
    return false;
}

// The triangle at place k of the pair list.
__device__ __forceinline__ int bin_triangle(const uint32_t *__restrict__ pairTri, int k, uint32_t triMask,
                                            int totalTris, Counters *ctr)
{
    const int tri = (int)(pairTri[k] & triMask);
    if ((unsigned)tri < (unsigned)totalTris) return tri;
    atomicOr(&ctr->errorFlags, (int)ERR_INTERNAL);
    return 0;
}

// Adds a warp's work counters to the launch's.
__device__ __forceinline__ void add_work(Counters *ctr, unsigned long long tested, uint32_t nrows, uint32_t npart,
                                         int lane)
{
    unsigned long long t = tested, tr = nrows, tp = npart;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        t += __shfl_xor_sync(kFullWarp, t, o);
        tr += __shfl_xor_sync(kFullWarp, tr, o);
        tp += __shfl_xor_sync(kFullWarp, tp, o);
    }
    if (lane == 0 && t) {
        atomicAdd(&ctr->pairTests, t);
        atomicAdd(&ctr->rowsEvaluated, tr);
        atomicAdd(&ctr->partialMasks, tp);
    }
}

// The ray-cast cross-check: a lane per sample of a bin, the warp streaming the
// bin's triangles through shared memory.  R: the row word (uint32_t for grids
// up to 32 x 32, u64 up to 64 x 64; a warp per block in the 64-bit form).  COUNT = 1: the work counters are
// accumulated (profiling).
template <class R, int COUNT>
__global__ void __launch_bounds__(RowWord<R>::kWarps * 32, RowWord<R>::kMinBlocks)
    k_raycast(const FrameDesc *__restrict__ frames, const FrameState *__restrict__ states,
              const int4 *__restrict__ items, int itemCapacity, Counters *ctr,
              const uint32_t *__restrict__ sortedVals, const int32_t *__restrict__ bss,
              const int32_t *__restrict__ bse, const int32_t *__restrict__ bts, const int32_t *__restrict__ bte,
              const uint32_t *__restrict__ pairTri, uint32_t triMask, const float4 *__restrict__ rec, int totalTris,
              int totalBins, int nframes)
{
    __shared__ StagedTri s_tri[RowWord<R>::kWarps][kOccChunk];
    __shared__ R s_rows[RowWord<R>::kWarps][RowWord<R>::kBits][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    R(*rows)[32] = s_rows[warp];
    StagedTri *tris = s_tri[warp];
    unsigned long long tested = 0;
    uint32_t nrows = 0;
    OccItem w;
    while (next_item(w, frames, items, itemCapacity, ctr, bss, bse, bts, bte, totalBins, nframes, sortedVals, lane)) {
        const FrameDesc &fr = frames[w.frame];
        const FrameState &st = states[w.frame];
        const GridC<R> g = grid_of<R>(fr);
        const f3 xd = ld3(fr.light.xd), yd = ld3(fr.light.yd), ur = ld3(fr.light.ur);
        const int chunk = chunk_of(fr);
        for (int first = w.sLo; first < w.sHi; first += 32) {
            LaneSample smp;
            int local = 0;
            R fullRows = g.FR;
            const bool has = item_sample(local, sortedVals, first + lane, w.sHi, fr, ctr);
            if (has) {
                load_sample(smp, fr, st, local);
                fullRows = init_rows<R>(fr, local, g, rows, lane);
            }
            for (int cur = 0; cur < w.nT && __any_sync(kFullWarp, fullRows != g.FR); cur += chunk) {
                const int m = min(chunk, w.nT - cur);
                __syncwarp();
                if (lane < m) stage_triangle(tris[lane], rec, bin_triangle(pairTri, w.tS + cur + lane, triMask, totalTris, ctr));
                __syncwarp();
                for (int t = 0; t < m; ++t) {
                    if (!__any_sync(kFullWarp, fullRows != g.FR)) break;
                    if (fullRows != g.FR) {
                        const int ts = raycast_pair<R, COUNT>(tris[t], smp, ur, xd, yd, g, rows, lane, fullRows, nrows);
                        if (COUNT) tested += ts;
                    }
                }
            }
            if (has) write_result<R>(fr, local, g, rows, lane);
        }
    }
    if (COUNT) add_work(ctr, tested, nrows, 0u, lane);
}


// ---------------------------------------------------------------------------
// k_occlusion_pairs: the same pair tests, scheduled so that every lane of a
// warp works on a pair that passed the AABB pre-cull.
//
// A warp owns a work item (up to 32 samples of one bin, one per lane, as in
// k_occlusion) and walks the bin's triangle list in chunks of kOccChunk staged
// triangles.  Per chunk:
//  1. cull: every lane tests its sample against each staged triangle's AABB and
//     minimum depth (the reference's pre-cull, K/Step5_2_shadowCalPerSample.inl
//     :120-128); a ballot per triangle gives the samples that pass it, and lane
//     t keeps the mask of triangle t;
//  2. compute: the passing pairs, numbered triangle-major through a warp scan
//     of the masks' popcounts, are dealt 32 at a time, one per lane; a lane
//     finds its pair's triangle by binary search over the scan, its sample as
//     the k-th set bit of that triangle's mask, fetches the sample's point from
//     the owning lane by shuffle and computes the pair's edge coefficients and
//     row filter;
//  3. rows: the (pair, light row) units of those 32 pairs are dealt 32 at a
//     time the same way; each lane evaluates the three row masks of its unit
//     (coefficients fetched from the pair's lane by shuffle) and ORs them into
//     the sample's row in shared memory by an atomic.
// A sample whose light rows are all full stops taking part (the reference's
// early-out); the pairs it still had in the chunk being dealt are skipped at
// their start.  The final mask is the OR over the bin's triangles either way.
// ---------------------------------------------------------------------------

#ifndef FDZB_OCC2_MINBLOCKS
#define FDZB_OCC2_MINBLOCKS 6
#endif

// Bit position of the k-th (0-based) set bit of m; k < popc(m).
__device__ __forceinline__ int nth_set_bit(uint32_t m, int k)
{
    int pos = 0;
    int c = __popc(m & 0xffffu);
    if (k >= c) { k -= c; pos += 16; m >>= 16; }
    c = __popc(m & 0xffu);
    if (k >= c) { k -= c; pos += 8; m >>= 8; }
    c = __popc(m & 0xfu);
    if (k >= c) { k -= c; pos += 4; m >>= 4; }
    c = __popc(m & 0x3u);
    if (k >= c) { k -= c; pos += 2; m >>= 2; }
    c = (int)(m & 1u);
    if (k >= c) pos += 1;
    return pos;
}

// The reference's row mask without branches: the threshold is computed
// whatever the case and selected away when the row is full or empty (the same
// mask as row_mask's).
__device__ __forceinline__ uint32_t row_mask_sel(float D, float slopeNm1, float slope, uint32_t full,
                                                 uint32_t &npart)
{
    const bool f1 = D >= 0.0f;
    const bool f2 = __fadd_rn(slopeNm1, D) >= 0.0f;
    const float q = __fdiv_rn(-D, slope);
    const int k = __float2int_ru(q);
    uint32_t m = ((unsigned)k >= 32u) ? 0u : (1u << k);
    m -= 1u;
    m = f1 ? m : ~m;
    npart += (f1 != f2) ? 1u : 0u;
    m = (f1 == f2) ? (f1 ? full : 0u) : m;
    return m & full;
}

// Edge coefficients of one pair (K/Step5_2_shadowCalPerSample.inl:129-191): the
// light rows still open after the row filter, or 0 (self-skip, or nothing).
struct PairEdges {
    float A[3], B[3], C[3], Bn[3];
};

__device__ __forceinline__ uint32_t pair_setup(const StagedTri &T, f3 Q, f3 L0Q, f3 xd, f3 yd, float esp,
                                               float nm1, uint32_t FULL, uint32_t fullRows, PairEdges &e,
                                               uint32_t &npart)
{
    const float4 p1 = T.p[1], p2 = T.p[2], p3 = T.p[3], p4 = T.p[4], p5 = T.p[5], p6 = T.p[6];
    const f3 v0 = mk3(p1.y, p1.z, p1.w), v1 = mk3(p2.x, p2.y, p2.z), v2 = mk3(p2.w, p3.x, p3.y);
    const f3 n = mk3(p3.z, p3.w, p4.x);
    const f3 e01 = mk3(p4.y, p4.z, p4.w), e12 = mk3(p5.x, p5.y, p5.z), e20 = mk3(p5.w, p6.x, p6.y);
    const float dir = dot3(sub3(Q, v0), n);
    if (fabsf(dir) < esp && point_in_tri(v0, v1, v2, Q)) return 0u;
    const bool neg = dir < 0.0f;
    const f3 t0 = neg ? mk3(-xd.x, -xd.y, -xd.z) : xd;
    const f3 t1 = neg ? mk3(-yd.x, -yd.y, -yd.z) : yd;
    const f3 lq = neg ? mk3(-L0Q.x, -L0Q.y, -L0Q.z) : L0Q;
    const f3 n0 = cross3(sub3(v1, Q), e01);
    const f3 n1 = cross3(sub3(v2, Q), e12);
    const f3 n2 = cross3(sub3(v0, Q), e20);
    e.A[0] = dot3(n0, t0); e.B[0] = dot3(n0, t1); e.C[0] = dot3(n0, lq);
    e.A[1] = dot3(n1, t0); e.B[1] = dot3(n1, t1); e.C[1] = dot3(n1, lq);
    e.A[2] = dot3(n2, t0); e.B[2] = dot3(n2, t1); e.C[2] = dot3(n2, lq);
    uint32_t vr = FULL & ~fullRows;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float An = __fmul_rn(e.A[k], nm1);
        e.Bn[k] = __fmul_rn(e.B[k], nm1);
        vr &= row_mask_sel(__fadd_rn(e.B[k] > 0.0f ? e.Bn[k] : 0.0f, e.C[k]), An, e.A[k], FULL, npart);
    }
    return vr;
}

__global__ void __launch_bounds__(kOccThreads, FDZB_OCC2_MINBLOCKS)
    k_occlusion_pairs(const FrameDesc *__restrict__ frames, const FrameState *__restrict__ states,
                      const int4 *__restrict__ items, int itemCapacity, Counters *ctr,
                      const uint32_t *__restrict__ sortedVals, const int32_t *__restrict__ bss,
                      const int32_t *__restrict__ bse, const int32_t *__restrict__ bts,
                      const int32_t *__restrict__ bte, const uint32_t *__restrict__ pairTri, uint32_t triMask,
                      const float4 *__restrict__ rec, int totalTris, int totalBins, int nframes)
{
    __shared__ StagedTri s_tri[kOccWarps][kOccChunk];
    __shared__ uint32_t s_rows[kOccWarps][kMaxLightN32][32];
    __shared__ uint32_t s_full[kOccWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t(*rows)[32] = s_rows[warp];
    volatile uint32_t *sfull = s_full[warp];
    StagedTri *tris = s_tri[warp];
    unsigned long long tested = 0, nexam = 0, nchunks = 0, nrounds = 0;
    uint32_t nrows = 0, npart = 0;
    int nitems = *(volatile const int *)&ctr->itemCount;
    if (nitems > itemCapacity) nitems = itemCapacity;

    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(&ctr->itemCursor, 1);
        it = __shfl_sync(kFullWarp, it, 0);
        if (it >= nitems) break;
        const int4 item = items[it];
        const int bin = item.x, fi = item.z;
        if ((unsigned)bin >= (unsigned)totalBins || (unsigned)fi >= (unsigned)nframes) {
            if (lane == 0) atomicOr(&ctr->errorFlags, (int)ERR_INTERNAL);
            continue;
        }
        const FrameDesc &fr = frames[fi];
        const FrameState &st = states[fi];
        const int S = fr.W * fr.H;
        const int sLo = bss[bin] + item.y;
        const int sHi = min(sLo + kItemSamples, bse[bin]);
        const int tS = bts[bin];
        const int nT = bte[bin] - tS;

        if (nT <= 0) {
            // no triangle in this bin: shadow 0 -- or, in a later triangle pass,
            // the result of the earlier passes, left as it is
            if (!fr.accumulate) {
                for (int k = sLo + lane; k < sHi; k += 32) {
                    const int local = (int)sortedVals[k] - fr.sampleBase;
                    if ((unsigned)local < (unsigned)S) write_zero(fr, local);
                    else atomicOr(&ctr->errorFlags, (int)ERR_INTERNAL);
                }
            }
            continue;
        }

        const int N = fr.light.N;
        const uint32_t FULL = fr.light.full;
        const float nm1 = (float)(N - 1);
        const f3 xd = ld3(fr.light.xd), yd = ld3(fr.light.yd);
        const float esp = fr.esp;

        LaneSample smp;
        smp.Q = mk3(0.f, 0.f, 0.f);
        smp.L0Q = smp.Q;
        smp.spx = smp.spy = smp.spz = smp.spw = smp.spZ = 0.f;
        int local = 0;
        bool has = false;
        {
            const int k = sLo + lane;
            if (k < sHi) {
                local = (int)sortedVals[k] - fr.sampleBase;
                if ((unsigned)local >= (unsigned)S) {
                    atomicOr(&ctr->errorFlags, (int)ERR_INTERNAL);
                } else {
                    has = true;
                    load_sample(smp, fr, st, local);
                }
            }
        }
        uint32_t fr0 = FULL;
        if (has) fr0 = init_rows<uint32_t>(fr, local, grid_of<uint32_t>(fr), rows, lane);
        else
            for (int r = 0; r < N; ++r) rows[r][lane] = 0u;
        sfull[lane] = fr0;
        bool active = has && fr0 != FULL;
        for (int base = 0; base < nT && __any_sync(kFullWarp, active); base += kOccChunk) {
            const int m = min(kOccChunk, nT - base);
            __syncwarp();
            if (lane < m) {
                int tri = (int)(pairTri[tS + base + lane] & triMask);
                if ((unsigned)tri >= (unsigned)totalTris) {
                    atomicOr(&ctr->errorFlags, (int)ERR_INTERNAL);
                    tri = 0;
                }
                stage_triangle(tris[lane], rec, tri);
            }
            __syncwarp();
            // 1. cull: lane t keeps the samples passing triangle t
            uint32_t mine = 0u;
            for (int t = 0; t < m; ++t) {
                const float4 p0 = tris[t].p[0];
                const float minz = tris[t].p[1].x;
                const bool pass = active && p0.x <= smp.spx && p0.y <= smp.spy && smp.spz <= p0.z &&
                                  smp.spw <= p0.w && minz <= smp.spZ;
                const uint32_t b = __ballot_sync(kFullWarp, pass);
                if (lane == t) mine = b;
            }
            // 2. compute: pairs numbered triangle-major
            nexam += (unsigned long long)m * (unsigned)__popc(__ballot_sync(kFullWarp, active));
            ++nchunks;
            const int cnt = __popc(mine);
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFullWarp, incl, o);
                if (lane >= o) incl += y;
            }
            const int total = __shfl_sync(kFullWarp, incl, 31);
            const int excl = incl - cnt;
            for (int p0 = 0; p0 < total; p0 += 32) {
                ++nrounds;
                // (a) one pair per lane: edge coefficients and open rows
                const int p = p0 + lane;
                int t = 0;
#pragma unroll
                for (int w = 16; w >= 1; w >>= 1) {
                    const int e = __shfl_sync(kFullWarp, excl, t + w);
                    if (e <= p) t += w;
                }
                const uint32_t mt = __shfl_sync(kFullWarp, mine, t);
                const int kth = p - __shfl_sync(kFullWarp, excl, t);
                const bool valid = p < total;
                const int sl = valid ? nth_set_bit(mt, kth) : lane;
                const f3 Q = mk3(__shfl_sync(kFullWarp, smp.Q.x, sl), __shfl_sync(kFullWarp, smp.Q.y, sl),
                                 __shfl_sync(kFullWarp, smp.Q.z, sl));
                const f3 L0Q = mk3(__shfl_sync(kFullWarp, smp.L0Q.x, sl), __shfl_sync(kFullWarp, smp.L0Q.y, sl),
                                   __shfl_sync(kFullWarp, smp.L0Q.z, sl));
                PairEdges pe;
#pragma unroll
                for (int k = 0; k < 3; ++k) pe.A[k] = pe.B[k] = pe.C[k] = pe.Bn[k] = 0.0f;
                uint32_t vr = 0u;
                if (valid) {
                    const uint32_t fullRows = sfull[sl];
                    if (fullRows != FULL) {
                        ++tested;
                        vr = pair_setup(tris[t], Q, L0Q, xd, yd, esp, nm1, FULL, fullRows, pe, npart);
                    }
                }
                // (b) the (pair, row) units of this round, one per lane
                const int uc = __popc(vr);
                int uin = uc;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(kFullWarp, uin, o);
                    if (lane >= o) uin += y;
                }
                const int utotal = __shfl_sync(kFullWarp, uin, 31);
                const int uex = uin - uc;
                for (int u0 = 0; u0 < utotal; u0 += 32) {
                    const int u = u0 + lane;
                    int j = 0;
#pragma unroll
                    for (int w = 16; w >= 1; w >>= 1) {
                        const int e = __shfl_sync(kFullWarp, uex, j + w);
                        if (e <= u) j += w;
                    }
                    const uint32_t vj = __shfl_sync(kFullWarp, vr, j);
                    const int kk = u - __shfl_sync(kFullWarp, uex, j);
                    const int slj = __shfl_sync(kFullWarp, sl, j);
                    float A[3], B[3], C[3], Bn[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        A[k] = __shfl_sync(kFullWarp, pe.A[k], j);
                        B[k] = __shfl_sync(kFullWarp, pe.B[k], j);
                        C[k] = __shfl_sync(kFullWarp, pe.C[k], j);
                        Bn[k] = __shfl_sync(kFullWarp, pe.Bn[k], j);
                    }
                    if (u < utotal) {
                        const int r = nth_set_bit(vj, kk);
                        ++nrows;
                        const float fr = (float)r;
                        uint32_t M = FULL;
#pragma unroll
                        for (int k = 0; k < 3; ++k)
                            M &= row_mask_sel(__fadd_rn(__fmul_rn(A[k], fr), C[k]), Bn[k], B[k], FULL, npart);
                        if (M) {
                            const uint32_t old = atomicOr(&rows[r][slj], M);
                            if (old != FULL && (old | M) == FULL) atomicOr((uint32_t *)&sfull[slj], 1u << r);
                        }
                    }
                }
            }
            __syncwarp();
            active = active && sfull[lane] != FULL;
        }
        __syncwarp();
        if (has) write_result<uint32_t>(fr, local, grid_of<uint32_t>(fr), rows, lane);
    }
    unsigned long long t = tested, tr = nrows, tp = npart;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        t += __shfl_xor_sync(kFullWarp, t, o);
        tr += __shfl_xor_sync(kFullWarp, tr, o);
        tp += __shfl_xor_sync(kFullWarp, tp, o);
    }
    if (lane == 0 && t) {
        atomicAdd(&ctr->pairTests, t);
        atomicAdd(&ctr->rowsEvaluated, tr);
        atomicAdd(&ctr->partialMasks, tp);
    }
    if (lane == 0 && nchunks) {
        atomicAdd(&ctr->pairsExamined, nexam);
        atomicAdd(&ctr->chunks, nchunks);
        atomicAdd(&ctr->rounds, nrounds);
    }
}

}  // namespace fdzb
