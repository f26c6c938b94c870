// warp_dev.cuh -- device helpers of the tricubic warp (S/ST_Tomo/warping.h:49-114):
// grid mapping, the CImg Catmull-Rom sampler with its 8-corner clamp, and the trace.
#pragma once

#include "stt_internal.cuh"

namespace stt {
namespace warpdev {

struct Dim3i {
    int x, y, z;
};

// world (aabb = [0,dim]) -> cell grid, clamped to [1, dim-2] (warping.h:54-62).
__device__ __forceinline__ float to_grid(float p, int dim, bool *clamped) {
    float gw = __fdiv_rn(__fmul_rn((float)dim, p), (float)dim);
    float gq = gw - 0.5f;
    const float hi = (float)(dim - 2), lo = 1.0f;
    bool c = !(gq >= lo && gq <= hi);
    gq = (gq < hi) ? gq : hi;  // std::min(hi, g)
    gq = (lo < gq) ? gq : lo;  // std::max(lo, g)
    if (clamped) *clamped = c;
    return gq;
}

// ---- forward sampler with 32-bit offsets and shared rows -------------------
// The grid coordinate g is already clamped to [1, dim-2], so with x = (int)g:
//  * taps x-1, x, x+1 are always inside the image.  CImg takes x instead of
//    x+1 when the fraction is 0, where the Catmull-Rom weight of that tap is
//    exactly 0: for finite data both give the same sum, and x+1 is then also
//    the cell's +1 corner, so the 8 corners are taps 1..2 on every axis and
//    need no loads of their own;
//  * tap x+2 leaves the image only when x = dim-2, i.e. g = dim-2 exactly and
//    the fraction is 0, where its weight is exactly 0: the tap is skipped
//    (a zero row or tap adds nothing), so no load ever leaves the image.
// I: the offsets inside a plane of voxels; long long is the general form, for 2^31
// voxels and more and for an axis of two voxels, which has x = 1, a fraction of 0 and
// no tap x+1: that form takes x for it (a weight of 0, and a corner already).
__host__ __device__ __forceinline__ bool needs_general(const Dim3i d) {
    return d.x < 3 || d.y < 3 || d.z < 3 || (long long)d.x * d.y * d.z >= (1LL << 31);
}

template <typename I>
struct Axis {
    I lo;        // element offset of tap 0 (x-1) along this axis
    I two;       // from it to tap 2 (the general form's)
    bool t3;     // tap 3 (x+2) inside the image
    float w[4];  // Catmull-Rom weights of the fraction
};

template <typename I>
__device__ __forceinline__ void axis_setup(float g, I stride, int dim, Axis<I> &a) {
    const int x = (int)g;
    cr_weights(g - (float)x, a.w);
    a.lo = (x - 1) * stride;
    a.two = x + 1 < dim ? 2 * stride : stride;
    a.t3 = x + 2 < dim;
}

template <typename I>
struct Cell {
    Axis<I> x, y, z;
    I sy, sz;  // row and plane strides
};

template <typename I>
__device__ __forceinline__ void cell_setup(const Dim3i d, const float g[3], Cell<I> &c) {
    c.sy = d.x;
    c.sz = (I)d.x * d.y;
    axis_setup<I>(g[0], 1, d.x, c.x);
    axis_setup(g[1], c.sy, d.y, c.y);
    axis_setup(g[2], c.sz, d.z, c.z);
}

// A tap: read-only global load (a BF16-stored image widened exactly), or a
// plain load when SHARED (img then points into shared memory, which the
// global read-only path cannot address).
// RW: a plain load of a global image that the running launch has written
// (the persistent iteration's Y_bc).
template <bool SHARED, typename T, bool RW = false>
__device__ __forceinline__ float ld_tap(const T *p) {
    if constexpr (SHARED) return *p;
    else if constexpr (RW) return ld_stored(p);
    else return ld_voxel(p);
}

// sample_image (warping.h:49-88) of NC planes that share one cell: the
// Catmull-Rom value of each, clamped to the min/max of its 8 cell corners.
// Plane p starts at img + p * pstride.  The sums run over x taps, then rows,
// then planes, contracted as written, so every kernel that samples rounds alike.
template <int NC, bool SHARED = false, typename T = float, bool RW = false, typename I = int>
__device__ __forceinline__ void sample_cell(const T *__restrict__ img, size_t pstride, const Cell<I> &s,
                                            float out[NC]) {
    constexpr bool GENERAL = sizeof(I) == 8;
    float val[NC], mn[NC], mx[NC];
#pragma unroll
    for (int p = 0; p < NC; ++p) {
        val[p] = 0.0f;
        mn[p] = INFINITY;
        mx[p] = -INFINITY;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (c == 3 && !s.z.t3) break;
        float yv[NC];
#pragma unroll
        for (int p = 0; p < NC; ++p) yv[p] = 0.0f;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            if (b == 3 && !s.y.t3) break;
            const I row = s.x.lo + s.y.lo + (GENERAL && b == 2 ? s.y.two : b * s.sy) + s.z.lo +
                          (GENERAL && c == 2 ? s.z.two : c * s.sz);
#pragma unroll
            for (int p = 0; p < NC; ++p) {
                const T *r = img + p * pstride + row;
                const float t0 = ld_tap<SHARED, T, RW>(r), t1 = ld_tap<SHARED, T, RW>(r + 1),
                            t2 = ld_tap<SHARED, T, RW>(r + (GENERAL ? s.x.two : 2));
                const float t3 = s.x.t3 ? ld_tap<SHARED, T, RW>(r + 3) : 0.0f;
                const float xv = __fmaf_rn(
                    s.x.w[3], t3, __fmaf_rn(s.x.w[2], t2, __fmaf_rn(s.x.w[0], t0, __fmul_rn(s.x.w[1], t1))));
                yv[p] = __fmaf_rn(s.y.w[b], xv, yv[p]);
                if ((b == 1 || b == 2) && (c == 1 || c == 2)) {
                    mn[p] = fminf(mn[p], fminf(t1, t2));
                    mx[p] = fmaxf(mx[p], fmaxf(t1, t2));
                }
            }
        }
#pragma unroll
        for (int p = 0; p < NC; ++p) val[p] = __fmaf_rn(s.z.w[c], yv[p], val[p]);
    }
#pragma unroll
    for (int p = 0; p < NC; ++p) out[p] = fmaxf(mn[p], fminf(val[p], mx[p]));
}

// The trace of voxel (i, j, k) through vel (warping.h:100-114) with step dt
// (the gather form's arithmetic: the exact centre read, the Catmull-Rom
// velocity sample at the half-traced point) and the cell of its end point.
template <typename I>
__device__ __forceinline__ void trace_cell(const Dim3i d, const float *__restrict__ vel, float dt, int i, int j,
                                           int k, Cell<I> &s) {
    const size_t n = (size_t)d.x * d.y * d.z;
    const float h = -dt;
    // cell centre (warping.h:25-29); the velocity there is an exact node read
    const float p[3] = {(float)i + 0.5f, (float)j + 0.5f, (float)k + 0.5f};
    const int ci = min(max(i, 1), d.x - 2), cj = min(max(j, 1), d.y - 2), ck = min(max(k, 1), d.z - 2);
    const I c = ci + (I)cj * d.x + (I)ck * d.x * d.y;
    const float v1[3] = {__ldg(vel + c), __ldg(vel + n + c), __ldg(vel + 2 * n + c)};
    // trace (warping.h:100-114): p2 = p + h v(p); p0 = p2 - h v(p2); q = p2 + (p - p0)/2
    float p2[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) p2[a] = __fadd_rn(p[a], __fmul_rn(h, v1[a]));
    const float g2[3] = {to_grid(p2[0], d.x, nullptr), to_grid(p2[1], d.y, nullptr),
                         to_grid(p2[2], d.z, nullptr)};
    Cell<I> s2;
    cell_setup(d, g2, s2);
    float v2[3];
    sample_cell<3>(vel, n, s2, v2);
    float q[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float p0 = __fsub_rn(p2[a], __fmul_rn(h, v2[a]));
        q[a] = __fadd_rn(p2[a], __fmul_rn(0.5f, __fsub_rn(p[a], p0)));
    }
    const float gq[3] = {to_grid(q[0], d.x, nullptr), to_grid(q[1], d.y, nullptr), to_grid(q[2], d.z, nullptr)};
    cell_setup(d, gq, s);
}

}  // namespace warpdev
}  // namespace stt
