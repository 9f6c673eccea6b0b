// fdzb_edge_masks.cuh -- k_occlusion, the edge-function row masks of a frame
// (stages c + d; K/Step5_2_shadowCalPerSample.inl:37-231).
//
// The reference decides a pair's light rows from its three edge functions in
// FP32: a row's mask is the columns [ceil lo, ceil hi) between the edges' zero
// crossings.  The crossings are where the edges of the triangle, projected from
// the sample onto the light's plane, cross the row, so a column's bit depends
// on the FP32 rounding only if a crossing lies within that rounding of an
// integer column.  The fast test below computes the crossings from the
// projected vertices -- a third of the reference's operations per pair and
// half per row -- together with a bound on how far the reference's own FP32
// crossings can be from its own; rows whose crossings stay clear of the integer
// columns by that bound are exactly the reference's, and the others (about one
// pair in a hundred) go through the reference's own operations (pair_test).
//
// Notation: light-grid coordinates of a point V are (X, Y, Z) with
// V = ur + X xd + Y yd + Z zn, zn the unit normal of the light's plane pointing
// at the scene; light sample (r, c) is (r, c, 0).  From the sample Q (depth
// h = Z_Q) a vertex at height dz = Z_Q - Z below the light's plane projects to
//   x = X_Q + (X - X_Q) t,  y = Y_Q + (Y - Y_Q) t,  t = h / dz.
// Every Y is kept half a column up (Y + 1/2), so that ceil(q) of a crossing q
// is the rounding to nearest of the value at hand.
//
// The bound, in columns (u = 2^-24; all distances world units; |.| lengths):
//  * the reference's crossing of an edge (a, b) over the whole grid.  Its
//    n = (b - Q) x (a - b) and the dot products with xd, yd and ur - Q are off
//    by at most 9.3 u |b - Q| |a - b| |.| in all (each operation's half ulp,
//    and the permanent of three vectors <= 2/sqrt(3) of their lengths'
//    product), so f(r, c) = A r + B c + C is off by 9.3 u |b - Q| |a - b| R,
//    R = |ur - Q| + rows |xd| + columns |yd|, and the crossing by that over
//    |B| = Vol dz_a dz_b |x_a - x_b| / h, Vol = |det(xd, yd, zn)|.  With
//    |b - Q| = dz_b |L - Q| / h, L the projected vertex, and P >= |L - Q|:
//    u 9.3 P R E t / (Vol h |x_a - x_b|), E the longest edge.
//  * the division's rounding and the comparisons at the grid's last column:
//    u 128; the reference's row filter, which must let through every row with
//    a clear crossing: u (64 + 192 |slope|) -- both small constants.
//  * the fast test's own: coordinates are rounded once (they are computed in
//    double), so x is off by u (6 t + 12) Sx, Sx = max(|X_Q|, |x|), and y
//    likewise; a line through two vertices inside their span is off by that in
//    y plus |slope| times that in x, and the rounding of its slope and constant
//    adds u (12 |slope| Sx + 2 Sy).
// So an edge with 1 / |x_a - x_b| = m is off by at most
//   t P k1 E m + |slope| ex + ey,  ex = u ((6 t + 24) Sx + 192),
//   ey = u ((6 t + 14) Sy + 128),
// with t, P, Sx, Sy the triangle's largest and every constant rounded up by 5 %
// or more.  In a row the long edge (between the extreme x) and the short edge
// of that row are active; the other short edge lies outside them by the row's
// distance from the middle vertex times the short edges' difference in slope,
// and rows beyond the triangle have the two edges crossed by the distance from
// that vertex times their difference in slope.  Where those exceed the bounds
// of the edges concerned at the nearest row (the computed slopes each off by at
// most 2 m times the edge's own part, and a line beyond its span by as much a
// row), they do so at every other row.  What is not clear by these bounds,
// after a closer look at the row concerned, goes to pair_test, as do vertices
// level with or below the sample, bounds of a quarter column or more, and
// triangles seen so nearly edge-on that the reference's side decision (the sign
// of dir) could differ (gs).
//
// Measured (B200, CUDA events, occlusion stage), against the reference's test
// for every pair with its quotients from hoisted reciprocals (the same masks), and
// after the steps noted below and the coverage order (k_tri_setup):
// 1920 x 1080 with 200k triangles, 16 x 16 light 5.33 -> 4.17 -> 2.95 ms, with 20k
// triangles 6.00 -> 3.61 -> 3.28 ms, 64 x 48 light 26.5 -> 19.7 -> 14.3 ms; 1280 x
// 720, 50k triangles up to and behind the light with the depth plane 25.3 -> 7.3 ->
// 6.70 ms; 3840 x 2160, 2M triangles, 32 x 32 light (whole frame) 1334 -> 382 -> 344 ms.
// Issue-bound (the first of these frames): 84 % of issue slots busy, the ALU pipe
// 66 %, 19.1 of 32 lanes.
#pragma once
#include "fdzb_occlusion.cuh"

namespace fdzb {

// A staged triangle: the four float4 of its fast record (k_tri_setup).
//  f0 = (aabb min x, min y, max x, max y)
//  f1 = (minz, E, X0, Y0)  f2 = (Z0, X1, Y1, Z1)  f3 = (X2, Y2, Z2, front)
// E: the longest edge, rounded up.  front: maxz of a triangle in front of the
// light's plane (minz > 0, every Z > 0), whose coordinates lie between the
// sample's and their projections; otherwise minus the largest |X| or |Y|.
struct FastTri {
    float4 f[4];
};

struct FastSample {
    float spx, spy, spz, spw, spZ;        // rectangle and depth (the pre-cull's)
    float X, Y, Z;                        // light-grid coordinates
    float P;                              // >= |ur - Q|
    float k1;                             // coefficient of E m in the bound
    float espK;                           // |dir| >= esp in units of the projected area's product
};

// Per-warp copy of the frame's constants (LightParams::fc).
enum FastConst { FC_SX = 0, FC_SY, FC_EXT, FC_KREF, FC_IVOL, FC_COUNT = 8 };
// Rows and columns by which the open-box cull widens a triangle: less leaves
// more triangles uncertain, more lets more of them through (1/64 to 1/2
// measured: 200k triangles 4.86, 4.56 at 1/8, 4.59 ms).
constexpr float kBoxMargin = 0.125f;
constexpr float kUlp = 1.0f / 16777216.0f;
constexpr float kErrT = 7.0f * kUlp, kErrX = 28.0f * kUlp, kErrY = 17.0f * kUlp;
constexpr float kErrRow = 256.0f * kUlp, kErrCol = 192.0f * kUlp;

__device__ __forceinline__ float rcp_approx(float b)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return y;
}
__device__ __forceinline__ float min3(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Warp-wide minimum / maximum of a float.
__device__ __forceinline__ float warp_min(float v)
{
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v)
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Light-grid coordinates of a point, computed in double and rounded once.
__device__ __forceinline__ f3 light_grid_coords(const LightParams &L, f3 v)
{
    const double x = (double)v.x - (double)L.ur[0], y = (double)v.y - (double)L.ur[1],
                 z = (double)v.z - (double)L.ur[2];
    return f3{(float)(L.G[0] * x + L.G[1] * y + L.G[2] * z), (float)(L.G[3] * x + L.G[4] * y + L.G[5] * z + 0.5),
              (float)(L.G[6] * x + L.G[7] * y + L.G[8] * z)};
}

// Coordinates for which nothing in either test overflows or underflows (the
// grid's steps are within [1e-8, 1e5], fdzb_light.cpp: grid_frame).
__device__ __forceinline__ bool in_range(f3 c)
{
    return fabsf(c.x) < 1e6f && fabsf(c.y) < 1e6f && fabsf(c.z) < 1e11f;
}

__device__ __forceinline__ void load_fast_sample(FastSample &s, const FrameDesc &fr, const FrameState &st, int local,
                                                 const float *fc)
{
    LaneSample ls;
    load_sample(ls, fr, st, local);
    s.spx = ls.spx;
    s.spy = ls.spy;
    s.spz = ls.spz;
    s.spw = ls.spw;
    s.spZ = ls.spZ;
    const f3 c = light_grid_coords(fr.light, ls.Q);
    s.X = c.x;
    s.Y = c.y;
    s.Z = c.z;
    const float d2 = ls.L0Q.x * ls.L0Q.x + ls.L0Q.y * ls.L0Q.y + ls.L0Q.z * ls.L0Q.z;
    s.P = sqrtf(d2) * 1.00001f;
    // a sample level with or behind the light, or out of range: no vertex counts
    // as above it, so every pair goes to pair_test
    if (!(c.z > 0.0f && in_range(c) && s.P < 1e11f)) s.Z = -__int_as_float(0x7f800000);
    s.k1 = fc[FC_KREF] * (s.P + fc[FC_EXT]) * rcp_approx(c.z);
    s.espK = fmaxf(fr.esp, 0.0f) * c.z * c.z * fc[FC_IVOL];
    if (isnan(fr.esp)) s.espK = fr.esp;   // every pair to self_skip
}

// Bits [a, b) of a row (none when b <= a), for a, b as 1.5 x 2^23 + integer,
// integer < 2^21.  NARROW: b - a is at most 31, so that the mask instruction's
// wrapping form takes the position from the float's low bits as they are.
constexpr float kIntBias = 12582912.0f;
template <class R, int NARROW> __device__ __forceinline__ R biased_range(float a, float b)
{
    const int width = max(__float_as_int(b) - __float_as_int(a), 0);
    uint32_t r;
    if constexpr (sizeof(R) == 8) {
        const uint32_t low = biased_range<uint32_t, 0>(a, b);
        const uint32_t high = biased_range<uint32_t, 0>(fmaxf(a, kIntBias + 32.0f) - 32.0f, b - 32.0f);
        return ((R)high << 32) | low;
    } else if constexpr (NARROW) {
        asm("bmsk.wrap.b32 %0, %1, %2;" : "=r"(r) : "r"(__float_as_int(a)), "r"(width));
    } else {
        asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(r) : "r"(__float_as_int(a) - __float_as_int(kIntBias)), "r"(width));
    }
    return r;
}

// Two FP32 values in one register pair: one instruction for both, each rounded as
// the scalar one.
struct Pair {
    u64 v;
};
__device__ __forceinline__ Pair pair_of(float a, float b)
{
    Pair p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(a), "f"(b));
    return p;
}
__device__ __forceinline__ void split(Pair p, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v));
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c)
{
    Pair d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return d;
}
__device__ __forceinline__ Pair add2(Pair a, Pair b)
{
    Pair d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}

template <class R>
__device__ __forceinline__ int highest_bit(R v)
{
    return (int)(8 * sizeof(R)) - 1 - (sizeof(R) == 8 ? __clzll((long long)v) : __clz((int)v));
}

// The reference's self-skip (K/Step5_2_shadowCalPerSample.inl:129-134).
__device__ __noinline__ bool self_skip(const float4 *__restrict__ rec, int tri, const float4 *__restrict__ pos, float esp)
{
    const float4 q0 = __ldg(rec + 4 * (size_t)tri), q1 = __ldg(rec + 4 * (size_t)tri + 1),
                 q2 = __ldg(rec + 4 * (size_t)tri + 2), P = __ldg(pos);
    const f3 v0 = mk3(q0.x, q0.y, q0.z), v1 = mk3(q1.x, q1.y, q1.z), v2 = mk3(q2.x, q2.y, q2.z);
    const f3 Q = mk3(P.x, P.y, P.z);
    const float dir = dot3(sub3(Q, v0), cross3(sub3(v1, v0), sub3(v2, v1)));
    return fabsf(dir) < esp && point_in_tri(v0, v1, v2, Q);
}

// The fast test of a triangle against the lane's sample.  Sets the rows it is
// certain of and returns the rows that pair_test has to decide (0 almost
// always).  BOX: a solid triangle (E > 0; see the open-box cull) that misses the
// open rows, or the columns [c0, c1] still open in some row, has no effect.
// With the depth plane, for triangles that reach the light's plane, the
// plane can only take bits away, so the rows that would gain one are left to
// pair_test -- unless the whole triangle is behind the light: a light sample
// in the projected triangle, with barycentric weights mu there, is on the far
// side of the triangle's plane where sum mu_i t_i >= 1, and every t_i < 1.  In
// FP32 the plane's value there is -|dir| (1 - sum mu t), off by at most
// 10 u E^2 (R + |v - Q|), and the edges' errors move sum mu t by at most
// 3 (10 u |v - Q| E R / |dir|) E / h_min.
template <class R, int DEPTH, int BOX, int COUNT, int NARROW>
__device__ __forceinline__ R fast_pair(const FastTri &T, const FastSample &s, const float *fc, float ncols, R FC,
                                       R open, float c0, float c1, R (*rows)[32], int lane, R &fullRows,
                                       uint32_t &nskip, uint32_t &tested, uint32_t &nrows, uint32_t &npart,
                                       const float4 *__restrict__ rec, const uint32_t *__restrict__ triAt,
                                       uint32_t triMask, int totalTris, const float4 *__restrict__ pos, float esp)
{
    constexpr float kRows = NARROW ? 16.0f : 64.0f;
    const float4 f1 = T.f[1], f2 = T.f[2], f3v = T.f[3];
    if (DEPTH && f3v.w >= s.spZ) return open;   // reaches the sample's depth: the plane counts
    const bool plane = DEPTH && f3v.w < 0.0f;
    const float dz0 = s.Z - f2.x, dz1 = s.Z - f2.w, dz2 = s.Z - f3v.z;
    const float i0 = rcp_approx(dz0), i1 = rcp_approx(dz1), i2 = rcp_approx(dz2);
    const float imin = min3(i0, i1, i2), imax = max3(i0, i1, i2), tm = s.Z * imax;
    if (!(imin > 0.0f && tm < 4096.0f)) {
        if (COUNT) ++tested;
        return open;   // a vertex level with or below the sample
    }
    const float t0 = s.Z * i0, t1 = s.Z * i1, t2 = s.Z * i2;
    const float y0 = __fmaf_rn(f1.w - s.Y, t0, s.Y), y1 = __fmaf_rn(f2.z - s.Y, t1, s.Y),
                y2 = __fmaf_rn(f3v.y - s.Y, t2, s.Y);
    const float x0 = __fmaf_rn(f1.z - s.X, t0, s.X), x1 = __fmaf_rn(f2.y - s.X, t1, s.X),
                x2 = __fmaf_rn(f3v.x - s.X, t2, s.X);
    const float ymin = min3(y0, y1, y2), ymax = max3(y0, y1, y2), ax = min3(x0, x1, x2), cx = max3(x0, x1, x2);
    if (BOX) {
        const float near = __fadd_ru(ax - kBoxMargin, kIntBias), far = __fadd_rd(cx + kBoxMargin, kIntBias + 1.0f);
        const R within = biased_range<R, NARROW>(fmaxf(near, kIntBias), fminf(far, kIntBias + kRows)) & open;
        if ((f1.y > 0.0f) & ((ymax < c0) | (ymin > c1) | (within == 0))) {
            ++nskip;
            return 0;
        }
    }
    if (COUNT) ++tested;
    // vertices by x: (ax, py), (bx, by), (cx, qy)
    float px = x0, py = y0, bx = x1, by = y1, qx = x2, qy = y2;
    {
        const bool sw = px > bx;
        const float u = sw ? bx : px, v = sw ? by : py;
        bx = sw ? px : bx;
        by = sw ? py : by;
        px = u;
        py = v;
    }
    {
        const bool sw = bx > qx;
        const float u = sw ? qx : bx, v = sw ? qy : by;
        qy = sw ? by : qy;
        bx = u;
        by = v;
    }
    {
        const bool sw = px > bx;
        const float v = sw ? by : py;
        bx = sw ? px : bx;
        by = sw ? py : by;
        py = v;
    }
    const float ay = py, cy = qy, w = cx - ax;
    const float mL = rcp_approx(w), m1 = rcp_approx(bx - ax), m2 = rcp_approx(cx - bx);
    const float aL = (cy - ay) * mL, a1 = (by - ay) * m1, a2 = (cy - by) * m2;
    const float kL = __fmaf_rn(-aL, ax, ay), k1 = __fmaf_rn(-a1, bx, by), k2 = __fmaf_rn(-a2, bx, by);
    // each edge's bound: m em + |slope| ex + ey
    const float xm = fmaxf(fabsf(ax), fabsf(cx)), ym = fmaxf(fabsf(ymin), fabsf(ymax));
    const float P = __fmaf_rn(xm, fc[FC_SX], __fmaf_rn(ym, fc[FC_SY], s.P));
    const float E = BOX ? fabsf(f1.y) : f1.y, em = tm * P * (s.k1 * E), tu = fmaxf(tm, 1.0f);
    const float ex = __fmaf_rn(max3(xm, fabsf(s.X), -f3v.w), __fmaf_rn(kErrT, tu, kErrX), kErrRow);
    const float ey = __fmaf_rn(max3(ym, fabsf(s.Y), -f3v.w), __fmaf_rn(kErrT, tu, kErrY), kErrCol);
    const float own1 = __fmaf_rn(fabsf(a1), ex, ey), own2 = __fmaf_rn(fabsf(a2), ex, ey), ownL = __fmaf_rn(fabsf(aL), ex, ey);
    const float errL = __fmaf_rn(mL, em, ownL), err1 = __fmaf_rn(m1, em, own1), err2 = __fmaf_rn(m2, em, own2);
    // half of what the edges' slopes may be off
    const float o1 = m1 * own1, o2 = m2 * own2, oL = mL * ownL;
    // the middle vertex's distance from the long edge, less what it may be off
    const float geo = by - __fmaf_rn(aL, bx, kL);
    const float gs = fabsf(geo) - errL * __fmaf_rn(2.0f * E, imax, 2.0f);
    // light rows inside [ax, cx] (first: rounded up, last: down) and at bx (down),
    // and the open ones among them
    const float b0 = __fadd_ru(ax, kIntBias), b1 = __fadd_rd(cx, kIntBias), bm = __fadd_rd(bx, kIntBias);
    const float fm = bx - (bm - kIntBias);
    R vr = biased_range<R, NARROW>(fmaxf(b0, kIntBias), fminf(b1, kIntBias + (kRows - 1.0f)) + 1.0f) & open;
    const int rFirst = RowWord<R>::lowest(vr), rLast = highest_bit<R>(vr);
    const float mid = max3((float)rFirst - bx, bx - (float)rLast, fminf(fm, 1.0f - fm));
    // the least differences of the slopes, and whether the nearest rows are clear
    const float dL1 = __fmaf_rn(-2.0f, oL + o1, fabsf(aL - a1)), dL2 = __fmaf_rn(-2.0f, oL + o2, fabsf(aL - a2));
    const float d12 = __fmaf_rn(-4.0f, o1 + o2, fabsf(a1 - a2));
    const float clear0 = __fmaf_rn((ax - (b0 - kIntBias)) + 1.0f, dL1, -(errL + err1));
    const float clear1 = __fmaf_rn((b1 - kIntBias) - cx + 1.0f, dL2, -(errL + err2));
    const float clearM = __fmaf_rn(mid, d12, -(err1 + err2));
    const float clearB = 0.0625f - ex * fmaxf(m1, m2);
    // the bounds of the edges that are active in some row
    float err = max3(errL, bm >= b0 ? err1 : 0.0f, bm < b1 ? err2 : 0.0f);
    R amb = 0;
    if (!(min3(min3(clear0, clear1, clearM), clearB, fminf(gs, 0.25f - errL)) > 0.0f)) {
        if (!(min3(clearB, gs, 0.25f - errL) > 0.0f)) return open;
        // At the row beyond an end the two edges' order is uncertain: that matters
        // only if the row is open and a column lies between them, give or take their
        // bounds; the next row must be clear.  Beside the middle vertex the short
        // edges are within their bounds of each other, which the row's bound covers.
        auto beyond = [&](float biasedRow, float a, float ka, float e) -> R {
            const float r = biasedRow - kIntBias, qa = __fmaf_rn(a, r, ka), qb = __fmaf_rn(aL, r, kL);
            const bool column = __fadd_rd(fmaxf(qa, qb) + e - 0.5f, kIntBias) >= __fadd_ru(fminf(qa, qb) - e - 0.5f, kIntBias);
            return column ? biased_range<R, 0>(fmaxf(biasedRow, kIntBias), biasedRow + 1.0f) & open : R(0);
        };
        const float eA = __fmaf_rn(1.0625f, errL + err1, 1e-6f), eC = __fmaf_rn(1.0625f, errL + err2, 1e-6f),
                    eB = __fmaf_rn(1.0625f, err1 + err2, 1e-6f);
        if (!(clear0 > 0.0f)) {
            if (!(dL1 > eA)) return open;
            amb |= beyond(b0 - 1.0f, a1, k1, eA);
        }
        if (!(clear1 > 0.0f)) {
            if (!(dL2 > eC)) return open;
            amb |= beyond(b1 + 1.0f, a2, k2, eC);
        }
        if (!(clearM > 0.0f)) {
            err = fmaxf(err, eB);
            if (!(d12 > 0.0f && err < 0.25f)) return open;
        }
    }
    // at most |dir| h^2 / Vol: beyond espK, |dir| is not below esp and nothing is skipped
    const float volume = dz0 * dz1 * dz2 * (w * gs);
    if (!(volume > s.espK)) {
        const int tri = (int)(*triAt & triMask);
        if ((unsigned)tri >= (unsigned)totalTris || self_skip(rec, tri, pos, esp)) return 0;
    }
    if (plane && tm < 1.0f) {
        const float tmin = s.Z * imin;
        if (volume * (0.9999f - tm) * tmin * s.Z > s.k1 * s.Z * s.Z * s.Z * E * E * (s.Z * tmin + 4.0f * P)) return 0;
    }
    if (!vr) return amb;
    const float thr = 0.5f - err;
    // the long edge is the lower one or the upper one: lower lines p, q and upper
    // lines u, v (one of the pairs twice the long edge)
    const bool lower = geo > 0.0f;
    const float ap = lower ? aL : a1, kp = lower ? kL : k1, aq = lower ? aL : a2, kq = lower ? kL : k2;
    const float au = lower ? a1 : aL, ku = lower ? k1 : kL, av = lower ? a2 : aL, kv = lower ? k2 : kL;
    R *row = &rows[rFirst][lane];
    R bit = R(1) << rFirst;
    // A row's cost is its issue slots, those of the integer and compare pipe most
    // (66 % of its rate at 84 % of the issue rate): the row number counts the loop, and
    // both ends are rounded as a pair.  1920 x 1080, 16 x 16 light: 4.15 -> 3.93 ms
    // (with a counter of its own 4.06; the lines as pairs too: 4.27).
    float rf = (float)rFirst;
    const Pair bias = pair_of(kIntBias, kIntBias), minus = pair_of(-1.0f, -1.0f);
    for (const float rl = (float)rLast; rf <= rl;) {
        const R have = *row;
        const float lo = max3(__fmaf_rn(ap, rf, kp), __fmaf_rn(aq, rf, kq), 0.0f);
        const float hi = min3(__fmaf_rn(au, rf, ku), __fmaf_rn(av, rf, kv), ncols);
        float bl, bh, dl, dh;
        const Pair ends = pair_of(lo, hi), rounded = add2(ends, bias);
        split(rounded, bl, bh);
        split(add2(ends, fma2(rounded, minus, bias)), dl, dh);   // the ends less the nearest integers
        const float off = fmaxf(fabsf(dl), fabsf(dh));
        R add = biased_range<R, NARROW>(bl, bh);
        if (COUNT) {
            ++nrows;
            npart += (lo > 0.0f) + (hi < ncols);
        }
        if (off > thr) {
            // the certain bits, and whether an uncertain one is still open
            const float e = __fmaf_rn(err, 1.0625f, 1e-6f);
            add = biased_range<R, 0>(fmaxf(lo + e, 0.0f) + kIntBias, fminf(hi - e, ncols) + kIntBias);
            const R may = biased_range<R, 0>(fmaxf(lo - e, 0.0f) + kIntBias, fminf(hi + e, ncols) + kIntBias);
            if (may & ~(add | have)) amb |= bit;
        }
        if (plane) {
            if (add & ~have) amb |= bit;
        } else {
            const R nv = have | add;
            *row = nv;
            if (nv == FC) fullRows |= bit;
        }
        row += 32;
        bit += bit;
        rf += 1.0f;
    }
    return amb & open;
}

// The reference's own test of triangle `tri` against sample `local`, for the
// rows in `open`.  Out of line: it is rare, and its registers would otherwise
// crowd the fast test's.  Returns the rows that are full now.
template <class R, int DEPTH, int COUNT>
__device__ __noinline__ R exact_pair(const FrameDesc &fr, const float4 *__restrict__ rec, int tri, int local,
                                     float spZ, R (*rows)[32], int lane, R open, R fullRows, Counters *ctr)
{
    const GridC<R> g = grid_of<R>(fr);
    uint32_t nrows = 0, npart = 0;
    StagedTri T;
    stage_triangle(T, rec, tri);
    const float4 P = __ldg(fr.pos + local);
    const f3 ur = ld3(fr.light.ur);
    LaneSample s;
    s.Q = mk3(P.x, P.y, P.z);
    s.L0Q = sub3(ur, s.Q);
    s.spZ = spZ;
    pair_test<R, DEPTH, COUNT>(T, s, ld3(fr.light.xd), ld3(fr.light.yd), ur, fr.esp, g, rows, lane, open, fullRows,
                               nrows, npart);
    if (COUNT) {
        atomicAdd(&ctr->rowsEvaluated, (unsigned long long)nrows);
        atomicAdd(&ctr->partialMasks, (unsigned long long)npart);
    }
    return fullRows;
}

// ---------------------------------------------------------------------------
// Open-box cull (BOX = 1).
//
// A triangle whose projection, widened by an eighth of a row and column, meets
// no unset bit of a sample sets none, and the mask -- the OR over the bin's
// triangles -- stays as it is without it.  When a chunk is staged, each lane
// tests one triangle for the whole warp: the columns still unset in some sample
// are OR-ed row by row, and the triangle is skipped if none lies in the
// rectangle that holds its projections from all of the warp's samples.  The
// projection of a vertex V,
//   x = (X_V Z_Q - X_Q Z_V) / (Z_Q - Z_V),
// is monotone in X_Q for a given Z_Q and in Z_Q for a given X_Q, so over the box of
// the samples its extremes are at the corners.  fast_pair repeats the test for
// the lane's own sample: against its open rows and the columns [c0, c1] unset in
// some row.
//
// The eighth covers the reference's FP32 edges: a light sample L that they
// accept has barycentric weights of at least -eps / (|dir| t) on the projected
// vertices (at most two of them negative), eps = 9.3 u D E R the edge functions'
// error, so it lies within 2 eps / (|dir| t) of the projected extent, itself at
// most t E (1 + t D / h), of that extent's box.  Triangles for
// which that may exceed an eighth for some sample of the warp -- seen nearly
// edge-on, or reaching down to the samples' depth -- are not culled (solid).
// ---------------------------------------------------------------------------
// The box of a warp's samples in light-grid coordinates, with their largest
// P, in shared memory.
struct SampleBox {
    float x, y, z, ex, ey, ez, P;   // centre, half sides, max P
    float spx, spy, spz, spw, spZ;  // the pre-cull's values that the most triangles pass
};

__device__ __forceinline__ SampleBox sample_box(const FastSample &s, bool has)
{
    const float inf = __int_as_float(0x7f800000);
    const float x0 = warp_min(has ? s.X : inf), x1 = warp_max(has ? s.X : -inf);
    const float y0 = warp_min(has ? s.Y : inf), y1 = warp_max(has ? s.Y : -inf);
    const float z0 = warp_min(has ? s.Z : inf), z1 = warp_max(has ? s.Z : -inf);
    return SampleBox{0.5f * (x0 + x1), 0.5f * (y0 + y1), 0.5f * (z0 + z1), 0.5001f * (x1 - x0), 0.5001f * (y1 - y0),
                     0.5001f * (z1 - z0), warp_max(has ? s.P : 0.0f), warp_max(has ? s.spx : -inf),
                     warp_max(has ? s.spy : -inf), warp_min(has ? s.spz : inf), warp_min(has ? s.spw : inf),
                     warp_max(has ? s.spZ : -inf)};
}

__device__ __forceinline__ bool solid(const FastTri &T, const SampleBox &b, const float *fc)
{
    const float4 f1 = T.f[1], f2 = T.f[2], f3v = T.f[3];
    const float low = b.z - b.ez, high = b.z + b.ez;
    const float dzmin = low - max3(f2.x, f2.w, f3v.z), dzmax = high - min3(f2.x, f2.w, f3v.z);
    const float tmax = high * rcp_approx(dzmin), tmin = low * rcp_approx(dzmax);
    const float ax = f2.y - f1.z, ay = f2.z - f1.w, az = f2.w - f2.x;
    const float bx = f3v.x - f1.z, by = f3v.y - f1.w, bz = f3v.z - f2.x;
    const float nx = ay * bz - az * by, ny = az * bx - ax * bz, nz = ax * by - ay * bx;
    const float dx = f1.z - b.x, dy = f1.w - b.y, dz = f2.x - b.z;
    const float dir = fabsf(nx * dx + ny * dy + nz * dz) - (fabsf(nx) * b.ex + fabsf(ny) * b.ey + fabsf(nz) * b.ez);
    const float E = f1.y;
    const float gx = (fabsf(dx) + b.ex) * fc[FC_SX], gy = (fabsf(dy) + b.ey) * fc[FC_SY], gz = fabsf(dz) + b.ez;
    const float D = sqrtf(gx * gx + gy * gy + gz * gz) + E;
    const float need = (20.0f / kBoxMargin) * kUlp * fc[FC_IVOL] * D * (b.P + fc[FC_EXT]) * E * E * tmax *
                       (1.0f + tmax * D * rcp_approx(low));
    return dzmin > 0.0f && low > 0.0f && dir * tmin * fminf(fc[FC_SX], fc[FC_SY]) > need;
}

// Whether a solid triangle's projections from the warp's samples can meet an
// unset bit of the warp's open rows.
template <class R>
__device__ __forceinline__ bool union_reach(const FastTri &T, const SampleBox &b, const R *open, int nrows)
{
    const float4 f1 = T.f[1], f2 = T.f[2], f3v = T.f[3];
    const float VX[3] = {f1.z, f2.y, f3v.x}, VY[3] = {f1.w, f2.z, f3v.y}, VZ[3] = {f2.x, f2.w, f3v.z};
    const float inf = __int_as_float(0x7f800000);
    float x0 = inf, x1 = -inf, y0 = inf, y1 = -inf;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float Z = k ? b.z + b.ez : b.z - b.ez;
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            const float t = Z * rcp_approx(Z - VZ[v]);
            const float xa = __fmaf_rn(VX[v] - (b.x - b.ex), t, b.x - b.ex), xb = __fmaf_rn(VX[v] - (b.x + b.ex), t, b.x + b.ex);
            const float ya = __fmaf_rn(VY[v] - (b.y - b.ey), t, b.y - b.ey), yb = __fmaf_rn(VY[v] - (b.y + b.ey), t, b.y + b.ey);
            x0 = min3(x0, xa, xb);
            x1 = max3(x1, xa, xb);
            y0 = min3(y0, ya, yb);
            y1 = max3(y1, ya, yb);
        }
    }
    // columns are half a column up: column c is at c + 1/2
    const int r0 = __float2int_ru(fmaxf(x0 - kBoxMargin, 0.0f)), r1 = min(__float2int_rd(fminf(x1 + kBoxMargin, 64.0f)), nrows - 1);
    const float c0 = __fadd_ru(fmaxf(y0 - (0.5f + kBoxMargin), 0.0f), kIntBias);
    const float c1 = __fadd_rd(fminf(y1 - (0.5f - kBoxMargin), 64.0f), kIntBias + 1.0f);
    const R cols = biased_range<R, 0>(c0, c1);
    R any = 0;
    for (int r = r0; r <= r1 && !any; ++r) any = open[r] & cols;
    return any != 0;
}

// The lane's open columns into c0, c1 (half a column up, widened by the margin),
// and the columns unset in some active lane's sample, row by row, into `open`.
template <class R>
__device__ __forceinline__ void open_bits(float &c0, float &c1, const GridC<R> &g, bool active, R (*rows)[32], int lane,
                                          R *open)
{
    R all = g.FC;
    for (int r = 0; r < g.NR; ++r) {
        const R v = rows[r][lane], o = active ? g.FC & ~v : R(0);
        all &= v;
        if constexpr (sizeof(R) == 8)
            open[r] = (R)__reduce_or_sync(kFullWarp, (uint32_t)o) | (R)__reduce_or_sync(kFullWarp, (uint32_t)(o >> 32)) << 32;
        else
            open[r] = __reduce_or_sync(kFullWarp, o);
    }
    const R ocol = g.FC & ~all;
    c0 = (float)RowWord<R>::lowest(ocol) + (0.5f - kBoxMargin);
    c1 = (float)highest_bit<R>(ocol) + (0.5f + kBoxMargin);
}

// Rows of a lane's sample that wait for the exact test, and the triangle's place in
// the pair list.  Four a lane, two with 64-bit rows (11 blocks still fit an SM):
// tests run for more lanes at once, and rows that others fill meanwhile need none
// (1920 x 1080, 200k triangles: 3.07 -> 3.02 ms; depth plane at 1280 x 720: 6.93 ->
// 6.74; resolved after each 32 triangles, as with one place: no gain).
template <class R> struct PendingRows {
    R rows;
    int at;
};
template <class R> constexpr int kPending = sizeof(R) == 8 ? 2 : 4;

// Blocks an SM: 8 for the 16-row form without the depth plane, whose 64 registers
// then spill little (1920 x 1080: 3.02 -> 2.97 ms, 16 mixed frames 25.7 -> 25.0 ms;
// 9 blocks 3.14); the depth plane's tests need more (6.74 ms at 7, 7.15 at 8).
// Teams get more registers (128 x 128 samples, 2000 triangles: 97 us a frame at 5,
// 107 at 7, 106 at 4).
template <class R, int DEPTH, int ROWS, int TEAM = 0>
constexpr int kOccBlocks = TEAM ? 5 : ROWS == 16 && !DEPTH ? 8 : RowWord<R>::kMinBlocks;

// Items an SM, at the most, of a launch that runs as teams; not the resident blocks,
// which take the items beyond them as they finish.  As teams / a warp an item, us a
// frame: 5.2 items an SM, 2000 triangles 105 / 142, 8000 167 / 347; 7.0 items, 400
// triangles 95 / 102, 8000 195 / 326.  Above the line teams still win at 9.1 items (8000
// triangles 208 / 398) and at 13.8 (2000: 121 / 140), and lose by far at 55 (the 480 x
// 270 view); where between is not measured.
constexpr int kTeamItems = 7;

// R: the row word (uint32_t for grids up to 32 x 32, u64 up to 64 x 64; a warp
// per block in the 64-bit form).
// DEPTH = 1: the pairs also test the triangle's own plane (pair_test).
// BOX = 1: the open-box cull.
// COUNT = 1: the work counters (pair tests, light rows, partial row masks) are
// accumulated; the engine runs this form when profiling is on.  The open-box
// cull's own counters (skipped and examined pairs) are kept in both forms.
// ROWS: light rows a lane's mask holds in shared memory (RowWord<R>::kBits, or
// 16 for launches whose grids have at most 16 rows of at most 31 columns).
// TEAM = 1: a block's warps take one item together, a chunk of its triangles
// each in turn, and OR their masks.  For launches of few items (kTeamItems), which
// last as long as their longest item: 128 x 96 samples, 400 triangles: 104 -> 94 us a
// frame.  With many items the warps do what an early-out of their own would have
// left out (480 x 270 of the dense frame: 1.7 ms, 6.2 as teams; 2.0 with masks
// exchanged every 16 triangles).
template <class R, int DEPTH, int BOX, int COUNT, int ROWS = RowWord<R>::kBits, int TEAM = 0>
__global__ void __launch_bounds__(RowWord<R>::kWarps * 32, kOccBlocks<R, DEPTH, ROWS, TEAM>)
    k_occlusion(const FrameDesc *__restrict__ frames, const FrameState *__restrict__ states,
                const int4 *__restrict__ items, int itemCapacity, Counters *ctr,
                const uint32_t *__restrict__ sortedVals, const int32_t *__restrict__ bss,
                const int32_t *__restrict__ bse, const int32_t *__restrict__ bts, const int32_t *__restrict__ bte,
                const uint32_t *__restrict__ pairTri, uint32_t triMask, const float4 *__restrict__ rec,
                const float4 *__restrict__ fastRec, int totalTris, int totalBins, int nframes)
{
    static_assert(ROWS >= 1 && ROWS <= RowWord<R>::kBits, "rows of a lane's mask");
    __shared__ FastTri s_tri[RowWord<R>::kWarps][kOccChunk];
    __shared__ R s_rows[RowWord<R>::kWarps][ROWS][32];
    __shared__ float s_fc[RowWord<R>::kWarps][FC_COUNT];
    __shared__ PendingRows<R> s_pend[RowWord<R>::kWarps][kPending<R>][32];
    __shared__ SampleBox s_box[BOX ? RowWord<R>::kWarps : 1];
    __shared__ R s_open[BOX ? RowWord<R>::kWarps : 1][BOX ? ROWS : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    R(*rows)[32] = s_rows[warp];
    FastTri *tris = s_tri[warp];
    const float *fc = s_fc[warp];
    unsigned long long boxSkips = 0, examined = 0, tested = 0;
    uint32_t nrows = 0, npart = 0;
    OccItem w;
    constexpr int kTeam = TEAM ? RowWord<R>::kWarps : 1;
    while (next_item<TEAM>(w, frames, items, itemCapacity, ctr, bss, bse, bts, bte, totalBins, nframes, sortedVals, lane)) {
        const FrameDesc &fr = frames[w.frame];
        const FrameState &st = states[w.frame];
        const GridC<R> g = grid_of<R>(fr);
        if (g.NR > ROWS || (ROWS == 16 && g.NC > 31)) {   // the host picks ROWS from the launch's largest grid
            if (lane == 0) atomicOr(&ctr->errorFlags, (int)ERR_INTERNAL);
            continue;   // in every warp of a team
        }
        __syncwarp();
        if (lane < FC_COUNT) s_fc[warp][lane] = fr.light.fc[lane];
        __syncwarp();
        // a team's warps take a chunk each in turn, shorter ones if the list is short
        const int chunk = TEAM ? min(chunk_of(fr), (w.nT + kTeam - 1) / kTeam) : chunk_of(fr);
        const float ncols = (float)g.NC;
        for (int first = w.sLo; first < w.sHi; first += 32) {
            FastSample smp;
            int local = 0;
            R fullRows = g.FR;
            const bool has = item_sample(local, sortedVals, first + lane, w.sHi, fr, ctr);
            if (has) {
                load_fast_sample(smp, fr, st, local, fc);
                fullRows = init_rows<R>(fr, local, g, rows, lane);
            }
            if (BOX) {
                const SampleBox b = sample_box(smp, has);
                if (lane == 0) s_box[warp] = b;
            }
            float c0 = 0.0f, c1 = 0.0f;
            // A lane's uncertain rows wait until some lane's places are taken, or the
            // list ends: the exact test then runs for every waiting lane at once, for
            // the rows that nothing else has filled.
            int waiting = 0;
            auto resolve = [&]() {
                for (int q = 0; __any_sync(kFullWarp, q < waiting && fullRows != g.FR); ++q) {
                    if (q < waiting && fullRows != g.FR) {
                        const PendingRows<R> p = s_pend[warp][q][lane];
                        const R todo = p.rows & ~fullRows;
                        if (todo)
                            fullRows = exact_pair<R, DEPTH, COUNT>(
                                fr, rec, bin_triangle(pairTri, p.at, triMask, totalTris, ctr), local, smp.spZ, rows, lane, todo,
                                fullRows, ctr);
                    }
                    __syncwarp();
                }
                waiting = 0;
            };
            for (int cur = TEAM ? warp * chunk : 0; cur < w.nT && __any_sync(kFullWarp, fullRows != g.FR);
                 cur += kTeam * chunk) {
                const int m = min(chunk, w.nT - cur);
                if (BOX) open_bits<R>(c0, c1, g, fullRows != g.FR, rows, lane, s_open[warp]);
                __syncwarp();
                bool mine = lane < m;
                if (mine) {
                    const int tri = bin_triangle(pairTri, w.tS + cur + lane, triMask, totalTris, ctr);
                    FastTri T;
#pragma unroll
                    for (int i = 0; i < 4; ++i) T.f[i] = __ldg(fastRec + 4 * (size_t)tri + i);
                    if (BOX) {
                        // the pre-cull for all of the warp's samples at once
                        const SampleBox &b = s_box[warp];
                        mine = T.f[0].x <= b.spx && T.f[0].y <= b.spy && b.spz <= T.f[0].z && b.spw <= T.f[0].w &&
                               T.f[1].x <= b.spZ;
                        if (!mine) {
                        } else if (!solid(T, s_box[warp], fc)) T.f[1].y = -T.f[1].y;
                        else mine = union_reach<R>(T, s_box[warp], s_open[warp], g.NR);
                    }
                    tris[lane] = T;
                }
                __syncwarp();
                unsigned keep = __ballot_sync(kFullWarp, mine);
                if (BOX && fullRows != g.FR) {
                    examined += (unsigned)m;
                    boxSkips += (unsigned)(m - __popc(keep));
                }
                for (; keep; keep &= keep - 1u) {
                    if (!__any_sync(kFullWarp, fullRows != g.FR)) break;
                    const int t = __ffs(keep) - 1;
                    if (fullRows != g.FR) {
                        const float4 f0 = tris[t].f[0];
                        if (f0.x <= smp.spx && f0.y <= smp.spy && smp.spz <= f0.z && smp.spw <= f0.w &&
                            tris[t].f[1].x <= smp.spZ) {
                            uint32_t skip = 0, ts = 0;
                            const int at = w.tS + cur + t;
                            const R open = g.FR & ~fullRows;
                            const R amb = fast_pair<R, DEPTH, BOX, COUNT, ROWS == 16>(
                                tris[t], smp, fc, ncols, g.FC, open, c0, c1, rows, lane, fullRows, skip, ts, nrows, npart, rec,
                                pairTri + at, triMask, totalTris, fr.pos + local, fr.esp);
                            if (BOX) boxSkips += skip;
                            if (COUNT) tested += ts;
                            if (amb) {
                                s_pend[warp][waiting][lane] = PendingRows<R>{amb, at};
                                ++waiting;
                            }
                        }
                    }
                    if (__any_sync(kFullWarp, waiting == kPending<R>)) resolve();
                }
            }
            if (__any_sync(kFullWarp, waiting > 0)) resolve();
            if (TEAM) {
                __syncthreads();
                if (warp == 0 && has) {
                    for (int r = 0; r < g.NR; ++r) {
                        R v = rows[r][lane];
#pragma unroll
                        for (int k = 1; k < kTeam; ++k) v |= s_rows[k][r][lane];
                        rows[r][lane] = v;
                    }
                    write_result<R>(fr, local, g, rows, lane);
                }
                if (first + 32 < w.sHi) __syncthreads();   // before the next samples' masks
            } else if (has) {
                write_result<R>(fr, local, g, rows, lane);
            }
        }
    }
    if (COUNT) add_work(ctr, tested, nrows, npart, lane);
    if (BOX) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            boxSkips += __shfl_xor_sync(kFullWarp, boxSkips, o);
            examined += __shfl_xor_sync(kFullWarp, examined, o);
        }
        if (lane == 0 && boxSkips) atomicAdd(&ctr->boxSkips, boxSkips);
        if (lane == 0 && examined) atomicAdd(&ctr->pairsExamined, examined);
    }
}

}  // namespace fdzb
