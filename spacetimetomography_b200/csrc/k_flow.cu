// k_flow.cu -- kernels of the 3D TV-L1/Huber optical flow of
// S/ST_Tomo/optical_flow.h (L1Huber_OF :83-623, L1Huber_OF_MultiScale3D
// :630-734) and of the CImg operations it calls (S/ImageFormationModel/CImg.h):
// the order-0 Deriche blur (deriche :32917-33050), resizing by moving average
// (:28135-28195) and by Catmull-Rom interpolation (:28432-28560), central
// differences with Neumann boundaries (get_gradient :34570-34581) and the
// warp of S/ST_Tomo/warping.h:49-145 over a general bounding box.
//
// This file is compiled with -fmad=false: every float and double expression
// is rounded operation by operation in the reference's order, so a level of
// the flow reproduces the reference's CPU result bit for bit (the residual
// sums, which the reference accumulates in a racy loop, are the exception).
//
// Layout: the caller's fields are planar and x-fastest, idx = x + y*nx +
// z*nx*ny, channel planes of n = nx*ny*nz floats (CImg's layout; dual field y: 10
// planes Y1|Y2|Y3|Y4).  The iterations work on vectors per voxel (Dual below),
// packed when a level starts.  Between residual checks one kernel runs the dual
// step of an iteration and the primal step of the next (k_flow_step).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>

#include "stt_kernels.h"

namespace stt {
namespace {

// std::min / std::max exactly as the reference calls them.
__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float smax(float a, float b) { return (a < b) ? b : a; }

struct Dims {
    int x, y, z;
};

__device__ __forceinline__ bool in_roi(const FlowRoi &r, const Dims &d, int i, int j, int k) {
    return k >= r.z0 && k < d.z - r.z1 && j >= r.y0 && j < d.y - r.y1 && i >= r.x0 && i < d.x - r.x1;
}

// ---- warp (warping.h:11-145) with aabb = [0, box] ---------------------------
// CImg::_cubic_atXYZ in its nested Catmull-Rom form (CImg.h:13429-13520): x
// rows first, then y, then z; taps clamped to the image, the "next" tap is
// x+1 only when the fraction is positive.
__device__ __forceinline__ float cimg_cr(float p, float c, float n, float a, float d) {
    return c + 0.5f * (d * (-p + n) + d * d * (2 * p - 5 * c + 4 * n - a) + d * d * d * (-p + 3 * c - 3 * n + a));
}

// Two of them in the packed FP32x2 instructions, each lane rounded as cimg_cr: a
// product is rounded on its own before it is added.  The compiler contracts packed
// products and sums whatever -fmad says, so a product is a fused multiply-add of a
// negative zero that it does not know (nz); doubling, quadrupling and halving are
// exact, so those products may stay fused.
__device__ __forceinline__ float2 cimg_cr2(float2 p, float2 c, float2 n, float2 a, float d, float nz) {
    const auto k = [](float x) { return make_float2(x, x); };
    const auto mul = [&](float x, float2 y) { return __ffma2_rn(k(x), y, k(nz)); };
    const auto sub = [&](float2 x, float2 y) { return __fadd2_rn(x, make_float2(-y.x, -y.y)); };
    const float2 c5 = mul(-5.0f, c);
    const float2 l = mul(d, sub(n, p));
    const float2 q = mul(d * d, sub(__ffma2_rn(k(4.0f), n, __ffma2_rn(k(2.0f), p, c5)), a));
    const float2 e = mul(d * d * d, __fadd2_rn(sub(sub(mul(3.0f, c), p), mul(3.0f, n)), a));
    return __ffma2_rn(k(0.5f), __fadd2_rn(__fadd2_rn(l, q), e), c);
}

// A world point's cell: the grid coordinate clamped to [1, dim-2], so taps x-1,
// x, x+1 are inside the image; CImg takes x for the tap x+1 where the fraction
// is zero, and the last voxel for x+2 past it.
struct BoxCell {
    int o[3];     // x, y, z of the first tap
    float d[3];   // fractions
    int last[3];  // the fourth tap, counted from the first: 3, or 2 at the upper edge
};

__device__ __forceinline__ void box_cell(const Dims &d, const float box[3], const float p[3], BoxCell &c) {
    const int D[3] = {d.x, d.y, d.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float q = (float)D[a] * (p[a] - 0.0f) / (box[a] - 0.0f) - 0.5f;
        const float hi = (float)(D[a] - 2), lo = 1.0f;
        q = (q < hi) ? q : hi;
        q = (lo < q) ? q : lo;
        const int x = (int)q;
        c.d[a] = q - (float)x;
        c.o[a] = x - 1;
        c.last[a] = x + 2 >= D[a] ? 2 : 3;
    }
}

// warping::sample_image: the cubic value clamped to the min/max of the cell's 8
// corners, which are taps of the stencil.  Rows go in pairs of planes.  I: the
// offsets inside a plane of voxels (int below 2^31 of them, else long long).
template <typename I>
__device__ __forceinline__ float sample_box(const float *__restrict__ img, const Dims &d, const BoxCell &q, float nz) {
    const I sy = d.x, sz = (I)d.x * d.y;
    const I at = q.o[0] + q.o[1] * sy + q.o[2] * sz;
    const float dx = q.d[0], dy = q.d[1], dz = q.d[2];
    float zv[4], corner[8];
#pragma unroll
    for (int c = 0; c < 4; c += 2) {
        float2 yv[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const I row = at + (b < 3 ? b : q.last[1]) * sy;
            const float *r0 = img + (row + c * sz), *r1 = img + (row + (c == 0 ? 1 : q.last[2]) * sz);
            const float2 t0 = make_float2(__ldg(r0), __ldg(r1)), t1 = make_float2(__ldg(r0 + 1), __ldg(r1 + 1));
            float2 t2 = make_float2(__ldg(r0 + 2), __ldg(r1 + 2));
            const float2 t3 = make_float2(__ldg(r0 + q.last[0]), __ldg(r1 + q.last[0]));
            if (b == 1 || b == 2) {  // planes 1 and 2 hold the corners: (x, y, z) at x + 2 y + 4 z
                const int m = 2 * (b - 1) + (c == 0 ? 0 : 4);
                corner[m] = c == 0 ? t1.y : t1.x;
                corner[m + 1] = c == 0 ? t2.y : t2.x;
            }
            if (!(dx > 0.0f)) t2 = t1;
            yv[b] = cimg_cr2(t0, t1, t2, t3, dx, nz);
        }
        if (!(dy > 0.0f)) yv[2] = yv[1];
        const float2 z = cimg_cr2(yv[0], yv[1], yv[2], yv[3], dy, nz);
        zv[c] = z.x, zv[c + 1] = z.y;
    }
    if (!(dz > 0.0f)) zv[2] = zv[1];
    const float val = cimg_cr(zv[0], zv[1], zv[2], zv[3], dz);
    constexpr int order[7] = {1, 3, 2, 4, 5, 7, 6};  // (the reference's, warping.h:71-80)
    float mn = corner[0], mx = mn;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        const float v = corner[order[k]];
        mn = (v < mn) ? v : mn;
        mx = (mx < v) ? v : mx;
    }
    const float inner = (val < mx) ? val : mx;
    return (mn < inner) ? inner : mn;
}

// warping::warp: trace back from each cell centre with -dt (two-step
// semi-Lagrangian, warping.h:100-114), sample every source channel there.  Seven
// samples of 64 taps and 21 uncontracted cubics a voxel: bound by issue.  So the
// three channels of a velocity share a cell, the corners of the clamp are taps, and
// ten of a sample's cubics are packed pairs.  One source channel, a cell and 21
// scalar cubics per sample in 64-bit offsets, blocks of 128 x 1 -> this, us: 54^3 126
// -> 53, 128^3 628 -> 300, 147 x 121 x 135 1289 -> 438, 256^3 5301 -> 2228 (scalar
// cubics 128^3 414; blocks of 32 x 4 in 168 registers 304, in 96 or 80 313).
constexpr int BOX_X = 32, BOX_Y = 8;
template <typename I>
__global__ void __launch_bounds__(BOX_X *BOX_Y, 2)
    k_warp_box(const Dims d, const float bx, const float by, const float bz, const float *__restrict__ vel,
               const float *__restrict__ src, int nc, float dt, float *__restrict__ out, float nz) {
    const int i = blockIdx.x * BOX_X + threadIdx.x;
    const int j = blockIdx.y * BOX_Y + threadIdx.y, k = blockIdx.z;
    if (i >= d.x || j >= d.y) return;
    const long long n = (long long)d.x * d.y * d.z;
    const float box[3] = {bx, by, bz};
    const int ijk[3] = {i, j, k};
    const int D[3] = {d.x, d.y, d.z};
    float p[3], v[3], p2[3], q[3];
    BoxCell cell;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (box[a] == (float)D[a])
            p[a] = (float)ijk[a] + 0.5f;  // (exactly what the division gives)
        else
            p[a] = (float)(0 + ((double)(float)ijk[a] + 0.5) * (double)(box[a] - 0) / (double)(float)D[a]);
    }
    const float h = -dt;
    box_cell(d, box, p, cell);
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] = sample_box<I>(vel + c * n, d, cell, nz);
#pragma unroll
    for (int c = 0; c < 3; ++c) p2[c] = p[c] + h * v[c];
    box_cell(d, box, p2, cell);
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] = sample_box<I>(vel + c * n, d, cell, nz);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float p0 = p2[c] - h * v[c];
        q[c] = p2[c] + 0.5f * (p[c] - p0);
    }
    box_cell(d, box, q, cell);
    const long long o = i + (long long)j * d.x + (long long)k * d.x * d.y;
    for (int c = 0; c < nc; ++c) out[o + c * n] = sample_box<I>(src + c * n, d, cell, nz);
}

// ---- per-warp setup (optical_flow.h:257-297) ---------------------------------
// Inside the ROI: the Neumann central gradient of the warped I2 and
// ut = I2w - I1 - grad.v.  Outside the ROI the reference leaves these arrays
// unset; here they are 0.  Everywhere: tau_c = 1/(4 + |u_c|) and
// sigma2 = 1/(|ux| + |uy| + |uz|) (infinite where the gradient vanishes).
// Before u is replaced, k4prev = u_prev . v keeps the data-term part of the
// previous warp's last K v, which the first dual step of this warp uses as
// its K v_old (the reference keeps Kx across warps, optical_flow.h:246, 394).
__global__ void __launch_bounds__(128) k_flow_setup(const Dims d, const FlowRoi roi, const float *__restrict__ i2w,
                                                    const float *__restrict__ i1, const float *__restrict__ v,
                                                    float4 *__restrict__ u, float4 *__restrict__ steps,
                                                    float *__restrict__ k4prev) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= d.x) return;
    const long long sy = d.x, sz = (long long)d.x * d.y, n = sz * d.z;
    const long long p = i + j * sy + k * sz;
    const float v1 = __ldg(v + p), v2 = __ldg(v + n + p), v3 = __ldg(v + 2 * n + p);
    const float4 up = u[p];
    k4prev[p] = up.x * v1 + up.y * v2 + up.z * v3;
    float ux = 0.0f, uy = 0.0f, uz = 0.0f, ut = 0.0f;
    if (in_roi(roi, d, i, j, k)) {
        const long long xm = i > 0 ? p - 1 : p, xp = i < d.x - 1 ? p + 1 : p;
        const long long ym = j > 0 ? p - sy : p, yp = j < d.y - 1 ? p + sy : p;
        const long long zm = k > 0 ? p - sz : p, zp = k < d.z - 1 ? p + sz : p;
        ux = (__ldg(i2w + xp) - __ldg(i2w + xm)) / 2;
        uy = (__ldg(i2w + yp) - __ldg(i2w + ym)) / 2;
        uz = (__ldg(i2w + zp) - __ldg(i2w + zm)) / 2;
        ut = __ldg(i2w + p) - __ldg(i1 + p) - ux * v1 - uy * v2 - uz * v3;
    }
    u[p] = make_float4(ux, uy, uz, ut);
    steps[p] = make_float4(1.0f / (4.0f / 1.0f + fabsf(ux)), 1.0f / (4.0f / 1.0f + fabsf(uy)),
                           1.0f / (4.0f / 1.0f + fabsf(uz)), 1.0f / (fabsf(ux) + fabsf(uy) + fabsf(uz)));
}

// The iterations' fields, a vector per voxel: a planar field costs a load and
// an address per float, and the step's 42 loads' addresses were most of its
// instructions.  v: (v1, v2, v3, unused) float4; u: (ux, uy, uz, ut); steps: (tau1,
// tau2, tau3, sigma2); y: n float4 (Y1x, Y1y, Y1z, Y2x), n float4 (Y2y, Y2z, Y3x,
// Y3y), n float2 (Y3z, Y4), one after the other.
struct Dual {
    float y[10];
};
// Chained launches overlap the one ahead: cached loads that are ordered after the
// wait, not the read-only path.
__device__ __forceinline__ float4 ld4(const float4 *p) { return __ldca(p); }
__device__ __forceinline__ Dual load_dual(const float *y, unsigned n, unsigned p) {
    const float4 *ya = reinterpret_cast<const float4 *>(y), *yb = ya + n;
    const float4 a = ld4(ya + p), b = ld4(yb + p);
    const float2 c = __ldca(reinterpret_cast<const float2 *>(yb + n) + p);
    return Dual{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y}};
}
__device__ __forceinline__ void store_dual(float *y, unsigned n, unsigned p, const float yn[9], float y4) {
    float4 *ya = reinterpret_cast<float4 *>(y), *yb = ya + n;
    ya[p] = make_float4(yn[0], yn[1], yn[2], yn[3]);
    yb[p] = make_float4(yn[4], yn[5], yn[6], yn[7]);
    reinterpret_cast<float2 *>(yb + n)[p] = make_float2(yn[8], y4);
}
__device__ __forceinline__ void spread(const float4 &a, float o[3]) { o[0] = a.x, o[1] = a.y, o[2] = a.z; }

// Start of a level: the caller's dual and flow packed; the flow into all three
// buffers (outside the ROI it is never updated).
__global__ void __launch_bounds__(256) k_flow_pack(unsigned n, const float *__restrict__ Y, const float *__restrict__ V,
                                                   float *__restrict__ y, float4 *__restrict__ v0,
                                                   float4 *__restrict__ v1, float4 *__restrict__ v2) {
    const unsigned p = blockIdx.x * 256 + threadIdx.x;
    if (p >= n) return;
    float q[10];
#pragma unroll
    for (int c = 0; c < 10; ++c) q[c] = __ldg(Y + (size_t)c * n + p);
    store_dual(y, n, p, q, q[9]);
    v0[p] = v1[p] = v2[p] =
        make_float4(__ldg(V + p), __ldg(V + (size_t)n + p), __ldg(V + (size_t)2 * n + p), 0.0f);
}

// Backward difference of S/ImageFormationModel/tools.cpp:146-192 (dxm3, dym3,
// dzm3) at coordinate c of n along a stride st, from the centre value a and
// the lower neighbour b (read only when c > 0): interior a - b, first a,
// last -b.
__device__ __forceinline__ float dm(float a, float b, int c, int n) {
    return (c > 0 && c < n - 1) ? a - b : (c == 0 ? a : -b);
}

// Forward difference of tools.cpp:126-138 (dxp3, dyp3, dzp3): upper
// neighbour b (read only when c < n-1) minus the centre a, 0 at the last.
__device__ __forceinline__ float dp(float a, float b, int c, int n) { return c < n - 1 ? b - a : 0.0f; }

// flags: bit 0 = residual iteration (iteration % 50 == 0); bit 1 = keep K^T y
// for the next iteration's residual; bit 2 = first iteration of the level
// (K v_old = 0, optical_flow.h:231-243); bit 3 = first iteration of a later
// warp (the data-term row of K v_old from k4prev).
constexpr int kResid = 1, kKeepKty = 2, kFirstOfLevel = 4, kFirstOfWarp = 8;

__device__ __forceinline__ void add_resid(double *resid, float r) {
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    if ((threadIdx.x & 31) == 0 && r != 0.0f) atomicAdd(resid, (double)r);
}

// Offsets inside one level are 32-bit: the host keeps 10 * voxels < 2^31.
// Every load of a voxel's neighbourhood is issued before the arithmetic.

// K^T y at one voxel (optical_flow.h:329-345): a: its dual, b: the lower
// neighbours' components (x, y, z of each flow component), u: the gradient.
__device__ __forceinline__ float kty_of(const float a[3], const float b[3], int i, int j, int k, const Dims &d, float u,
                                        float y4) {
    // -stepsizeD * dxm3 - ... with unit step sizes: (-1 * x) == -x and 1 * x == x exactly
    return -dm(a[0], b[0], i, d.x) - dm(a[1], b[1], j, d.y) - dm(a[2], b[2], k, d.z) + u * y4;
}

// Primal step over the ROI (optical_flow.h:314-370):
// Kty_c = -div_b(y_c) + u_c*y4; v_c -= tau_c*Kty_c, read from v_in and
// written to v_out (the dual step needs both).
__global__ void __launch_bounds__(128) k_flow_primal(const Dims d, const FlowRoi roi, const float *__restrict__ y,
                                                     const float4 *__restrict__ u, const float4 *__restrict__ steps,
                                                     const float4 *__restrict__ v_in, float4 *__restrict__ v_out,
                                                     float *__restrict__ kty, int flags, double *__restrict__ resid,
                                                     const int *__restrict__ done) {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    if (__ldca(done)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    float pr = 0.0f;
    if (i < d.x && in_roi(roi, d, i, j, k)) {
        const unsigned sy = d.x, sz = d.x * d.y, n = sz * d.z;
        const unsigned p = i + j * sy + k * sz;
        const Dual a = load_dual(y, n, p), bx = load_dual(y, n, i > 0 ? p - 1 : p);
        const Dual by = load_dual(y, n, j > 0 ? p - sy : p), bz = load_dual(y, n, k > 0 ? p - sz : p);
        const float4 up = ld4(u + p), vp = ld4(v_in + p), sp = ld4(steps + p);
        float uc[3], vo[3], t[3], vn[3];
        spread(up, uc), spread(vp, vo), spread(sp, t);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float b[3] = {bx.y[3 * c], by.y[3 * c + 1], bz.y[3 * c + 2]};
            const float kt = kty_of(a.y + 3 * c, b, i, j, k, d, uc[c], a.y[9]);
            vn[c] = vo[c] - t[c] * kt;
            if (flags & kResid) {
                const float r = fabsf((vo[c] - vn[c]) / t[c] - __ldca(kty + p + (size_t)c * n) + kt);
                pr = c == 0 ? r : pr + r;
            }
            if (flags & kKeepKty) kty[p + (size_t)c * n] = kt;
        }
        v_out[p] = make_float4(vn[0], vn[1], vn[2], 0.0f);
    }
    if (flags & kResid) add_resid(resid, pr);
}

// Constants of the dual step; lam2_lo: a bound just below lambda^2.
struct DualPar {
    float sigma1, hf, lambda, lam2_lo;
    int huber;
};

// One flow component's dual (optical_flow.h:394-470): the ascent
// yo + sigma1 (2 K v - K v_old), scaled by the Huber factor, projected onto the
// lambda-ball.
__device__ __forceinline__ void dual_channel(const float yo[3], const float kn[3], const float ko[3], const DualPar &q,
                                             float yn[3]) {
    float yt[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float t = yo[a] + q.sigma1 * (kn[a] + kn[a] - ko[a]);
        yt[a] = q.huber ? t * q.hf : t;
    }
    // divisor = max(1, sqrt(s)/lambda) and y = yt/divisor.  Below lam2_lo
    // (< lambda^2 with margin) sqrt(s) rounds below lambda, so the divisor is
    // exactly 1 and y = yt exactly: skip the sqrt and the divisions.
    const float ss = yt[0] * yt[0] + yt[1] * yt[1] + yt[2] * yt[2];
    yn[0] = yt[0], yn[1] = yt[1], yn[2] = yt[2];
    if (!(ss < q.lam2_lo)) {
        const float div = smax(1.0f, sqrtf(ss) / q.lambda);
        if (div != 1.0f) {
            yn[0] = yt[0] / div;
            yn[1] = yt[1] / div;
            yn[2] = yt[2] / div;
        }
    }
}

// Dual step over every voxel (optical_flow.h:374-497): K v by forward
// differences of v and u.v; over-relaxed ascent y + sigma1*(2 K v - K v_old),
// scaled by the Huber factor for norm 4; each y_c projected onto the
// lambda-ball; y4 clamped to [-1, 1].  K v_old, which the reference stores
// (10 floats per voxel), is recomputed here from v_old with the same float
// operations, so it is the same value.
__global__ void __launch_bounds__(128) k_flow_dual(const Dims d, const float4 *__restrict__ v,
                                                   const float4 *__restrict__ v_old, const float4 *__restrict__ u,
                                                   const float4 *__restrict__ steps, const float *__restrict__ k4prev,
                                                   float *__restrict__ y, const DualPar q, int flags,
                                                   double *__restrict__ resid, const int *__restrict__ done) {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    if (__ldca(done)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    float dr = 0.0f;
    if (i < d.x) {
        const unsigned sy = d.x, sz = d.x * d.y, n = sz * d.z;
        const unsigned p = i + j * sy + k * sz;
        const unsigned ox = i < d.x - 1 ? 1 : 0, oy = j < d.y - 1 ? sy : 0, oz = k < d.z - 1 ? sz : 0;
        const bool zero_old = flags & kFirstOfLevel;
        const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float vc[3], vx[3], vy[3], vz[3], oc[3], oxv[3], oyv[3], ozv[3];
        spread(ld4(v + p), vc), spread(ld4(v + p + ox), vx), spread(ld4(v + p + oy), vy), spread(ld4(v + p + oz), vz);
        spread(zero_old ? zero : ld4(v_old + p), oc), spread(zero_old ? zero : ld4(v_old + p + ox), oxv);
        spread(zero_old ? zero : ld4(v_old + p + oy), oyv), spread(zero_old ? zero : ld4(v_old + p + oz), ozv);
        const float4 *ya = reinterpret_cast<const float4 *>(y), *yb = ya + n;
        const float4 y0 = ld4(ya + p), y1 = ld4(yb + p);
        const float2 y2 = __ldca(reinterpret_cast<const float2 *>(yb + n) + p);
        const float yo[10] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w, y2.x, y2.y};
        const float4 up = ld4(u + p);
        const float s2 = ld4(steps + p).w;
        float yn[9];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            // K v with unit step sizes (stepsizeD = 1: x * 1.0f == x, dropped)
            const float kn[3] = {dp(vc[c], vx[c], i, d.x), dp(vc[c], vy[c], j, d.y), dp(vc[c], vz[c], k, d.z)};
            const float ko[3] = {dp(oc[c], oxv[c], i, d.x), dp(oc[c], oyv[c], j, d.y), dp(oc[c], ozv[c], k, d.z)};
            dual_channel(yo + 3 * c, kn, ko, q, yn + 3 * c);
            if (flags & kResid) {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const float r = fabsf((yo[3 * c + a] - yn[3 * c + a]) / q.sigma1 - ko[a] + kn[a]);
                    dr = (c == 0 && a == 0) ? r : dr + r;
                }
            }
        }
        const float k4 = up.x * vc[0] + up.y * vc[1] + up.z * vc[2];
        float k4o = 0.0f;
        if (flags & kFirstOfWarp) k4o = __ldca(k4prev + p);
        else if (!zero_old) k4o = up.x * oc[0] + up.y * oc[1] + up.z * oc[2];
        const float y4 = smax(-1.0f, smin(1.0f, yo[9] + s2 * (k4 + k4 - k4o + up.w)));
        store_dual(y, n, p, yn, y4);
        if (flags & kResid) dr = dr + fabsf((yo[9] - y4) / s2 - k4o + k4);
    }
    if (flags & kResid) add_resid(resid + 1, dr);
}

// The dual step of one iteration and the primal step of the next in one pass
// (neither a residual iteration): y_in -> y_out and (v, v_old) -> v_next.  The
// primal step at a voxel needs the new dual at the voxel and one voxel down each
// axis.  A block owns 31 x STEP_Y columns and walks up z: lane 0 and row 0 are
// the neighbouring columns' duals, formed here again (and not written); the
// x neighbour's comes from the lane below, the y neighbour's through shared
// memory, the z neighbour's from the step before.  The next plane's loads are in
// flight during the exchange and the stores.  y and v_next have buffers of their
// own: neighbouring blocks read the old ones.  The operations are the two
// kernels', so are the bits.
//
// An iteration moves 160 bytes per voxel where the two kernels moved 212, in one
// launch.  The next step's blocks come up while this one's last ones finish
// (launch_chained; they are let up two planes before a block's end: from its
// start they take the places that the last round's blocks spread over, 256^3 538
// -> 555).  Per iteration, two planar kernels -> this -> chained, us: 54^3 14.7 ->
// 8.8, 48^3 10.7 -> 8.7 -> 6.9, 80^3 23.5 -> 17.6 -> 16.5, 128^3 79.1 -> 76.0 ->
// 70.7, 147 x 121 x 135 110.6 -> 88.9 -> 81.9, 256^3 606 -> 538 -> 528 (5.1 TB/s).
// Bound by the latency of a plane's chain (loads, duals, exchange) at 20 warps
// per SM; so small blocks, whose barriers hold fewer warps up, beat the smaller
// halo of larger ones (unchained, STEP_Y 8, two blocks: 80 us at 128^3; 12: 80;
// 16: 92).  Measured and not kept: planar fields (42 loads and their addresses a
// voxel: 82), planes through a shared-memory ring by asynchronous copies (83),
// one component at a time in 72 registers (94), the steps formed from u instead
// of read (four divisions: 79).
constexpr int STEP_Y = 4;
__global__ void __launch_bounds__(32 * (STEP_Y + 1), 4)
    k_flow_step(const Dims d, const FlowRoi roi, const float *__restrict__ y_in, float *__restrict__ y_out,
                const float4 *__restrict__ v, const float4 *__restrict__ v_old, float4 *__restrict__ v_next,
                const float4 *__restrict__ u, const float4 *__restrict__ steps, const float *__restrict__ k4prev,
                float *__restrict__ kty, const DualPar q, int flags, int planes, const int *__restrict__ done) {
    __shared__ float below[2][STEP_Y + 1][3][32];
    cudaGridDependencySynchronize();
    if (__ldca(done)) return;
    const int lane = threadIdx.x, row = threadIdx.y;
    const int i0 = (int)blockIdx.x * 31 + lane - 1, j0 = (int)blockIdx.y * STEP_Y + row - 1;
    const bool own = lane > 0 && row > 0 && i0 < d.x && j0 < d.y;
    const int i = min(max(i0, 0), d.x - 1), j = min(max(j0, 0), d.y - 1);
    const unsigned sy = d.x, sz = d.x * d.y, n = sz * d.z;
    const unsigned ox = i < d.x - 1 ? 1 : 0, oy = j < d.y - 1 ? sy : 0;
    const int z0 = blockIdx.z * planes, z1 = min(z0 + planes, d.z);
    const bool zero_old = flags & kFirstOfLevel;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int k = z0 > 0 ? z0 - 1 : 0;
    unsigned p = i + j * sy + k * sz;
    float4 vc = ld4(v + p), oc = zero_old ? zero : ld4(v_old + p), vx, vy, vz, oxv = zero, oyv = zero, ozv = zero, up, sp;
    float pz[3] = {0.0f, 0.0f, 0.0f};
    Dual yo;
    // everything the dual step reads at offset o of plane kk but its own v and v_old
    auto load = [&](int kk, unsigned o) {
        const unsigned oz = kk < d.z - 1 ? sz : 0;
        vx = ld4(v + o + ox), vy = ld4(v + o + oy), vz = ld4(v + o + oz);
        if (!zero_old) oxv = ld4(v_old + o + ox), oyv = ld4(v_old + o + oy), ozv = ld4(v_old + o + oz);
        yo = load_dual(y_in, n, o);
        up = ld4(u + o);
        sp = ld4(steps + o);
    };
    load(k, p);
    for (int buf = 0; k < z1; ++k, p += sz, buf ^= 1) {
        if (k + 2 >= z1) cudaTriggerProgrammaticLaunchCompletion();
        const bool mine = own && k >= z0;
        const bool inside = mine && in_roi(roi, d, i, j, k);
        float a[3], bx[3], by[3], bz[3], e[3], fx[3], fy[3], fz[3], yn[9], xm[3];
        spread(vc, a), spread(vx, bx), spread(vy, by), spread(vz, bz);
        spread(oc, e), spread(oxv, fx), spread(oyv, fy), spread(ozv, fz);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float kn[3] = {dp(a[c], bx[c], i, d.x), dp(a[c], by[c], j, d.y), dp(a[c], bz[c], k, d.z)};
            const float ko[3] = {dp(e[c], fx[c], i, d.x), dp(e[c], fy[c], j, d.y), dp(e[c], fz[c], k, d.z)};
            dual_channel(yo.y + 3 * c, kn, ko, q, yn + 3 * c);
            xm[c] = __shfl_up_sync(0xffffffffu, yn[3 * c], 1);
            below[buf][row][c][lane] = yn[3 * c + 1];
        }
        const float k4 = up.x * a[0] + up.y * a[1] + up.z * a[2];
        float k4o = 0.0f;
        if (flags & kFirstOfWarp) k4o = __ldca(k4prev + p);
        else if (!zero_old) k4o = up.x * e[0] + up.y * e[1] + up.z * e[2];
        const float y4 = smax(-1.0f, smin(1.0f, yo.y[9] + sp.w * (k4 + k4 - k4o + up.w)));
        float uc[3], t[3];
        spread(up, uc), spread(sp, t);
        vc = vz, oc = ozv;
        if (k + 1 < z1) load(k + 1, p + sz);  // the next plane's loads fly during the exchange and the stores
        __syncthreads();  // (the other buffer is read before this plane's barrier, written after it)
        if (mine) {
            store_dual(y_out, n, p, yn, y4);
            if (inside) {
                float vn[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float b[3] = {xm[c], below[buf][row - 1][c][lane], pz[c]};
                    const float kt = kty_of(yn + 3 * c, b, i, j, k, d, uc[c], y4);
                    vn[c] = a[c] - t[c] * kt;
                    if (flags & kKeepKty) kty[p + (size_t)c * n] = kt;
                }
                v_next[p] = make_float4(vn[0], vn[1], vn[2], 0.0f);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) pz[c] = yn[3 * c + 2];
    }
}

// End of a warp: the flow of the last iteration that ran lies in buffer
// iters % 3; unpack it into the caller's planes, and bring it to the first
// buffer for the next warp.
__global__ void __launch_bounds__(256) k_flow_settle(unsigned n, const int *__restrict__ iters,
                                                     const float4 *__restrict__ v_1, const float4 *__restrict__ v_2,
                                                     float4 *__restrict__ v_0, float *__restrict__ V) {
    const unsigned p = blockIdx.x * 256 + threadIdx.x;
    if (p >= n) return;
    const int at = *iters % 3;
    const float4 r = at == 0 ? v_0[p] : ld4((at == 1 ? v_1 : v_2) + p);
    if (at != 0) v_0[p] = r;
    V[p] = r.x;
    V[(size_t)n + p] = r.y;
    V[(size_t)2 * n + p] = r.z;
}

// Stopping rule of optical_flow.h:306, 488-491: after a residual iteration
// err = (d^2 + p^2)/n, and the loop stops unless err > tol.  Records the
// iteration count of the warp (when it stops, or at the last iteration).
__global__ void k_flow_check(double *resid, long long n, float tol, int it, int is_resid, int is_last, int *done,
                             int *iters, float *err) {
    if (*done) return;
    if (is_resid) {
        const float pf = (float)resid[0], df = (float)resid[1];
        const float e = (df * df + pf * pf) / (float)n;
        *err = e;
        resid[0] = 0.0;
        resid[1] = 0.0;
        if (!(e > tol)) {
            *done = 1;
            *iters = it;
            return;
        }
    }
    if (is_last) *iters = it;
}

// Start of a warp: clear the stop flag and the residual sums, reset the
// iteration count and set the recorded residual to its initial value 1.
__global__ void k_flow_reset(int *done, double *resid, int *iters, float *err) {
    *done = 0;
    resid[0] = 0.0;
    resid[1] = 0.0;
    *iters = 0;
    *err = 1.0f;
}

// ---- CImg::deriche, order 0, Neumann (CImg.h:32917-33050) ---------------------
// One thread per line along `axis`, in place; the causal pass is buffered in
// `tmp` at the same positions.
__global__ void k_deriche_line(const Dims d, int nc, int axis, const DericheCoef c, float *__restrict__ img,
                               float *__restrict__ tmp) {
    const long long per_ch = axis == 0 ? (long long)d.y * d.z : axis == 1 ? (long long)d.x * d.z : (long long)d.x * d.y;
    const long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (l >= per_ch * nc) return;
    const long long n3 = (long long)d.x * d.y * d.z;
    const int ch = (int)(l / per_ch);
    const long long r = l % per_ch;
    long long base, off;
    int N;
    if (axis == 0) {
        N = d.x;
        off = 1;
        base = r * d.x;
    } else if (axis == 1) {
        N = d.y;
        off = d.x;
        base = (r % d.x) + (r / d.x) * (long long)d.x * d.y;
    } else {
        N = d.z;
        off = (long long)d.x * d.y;
        base = r;
    }
    float *X = img + ch * n3 + base;
    float *Y = tmp + ch * n3 + base;
    float xp = X[0], yb = c.coefp * xp, yp = yb;
    for (int m = 0; m < N; ++m) {
        const float xc = X[m * off];
        const float yc = c.a0 * xc + c.a1 * xp - c.b1 * yp - c.b2 * yb;
        Y[m * off] = yc;
        xp = xc;
        yb = yp;
        yp = yc;
    }
    float xn = X[(N - 1) * off], xa = xn, yn = c.coefn * xn, ya = yn;
    for (int m = N - 1; m >= 0; --m) {
        const float xc = X[m * off];
        const float yc = c.a2 * xn + c.a3 * xa - c.b1 * yn - c.b2 * ya;
        xa = xn;
        xn = xc;
        ya = yn;
        yn = yc;
        X[m * off] = Y[m * off] + yc;
    }
}

// ---- CImg::get_resize(..., 5), one axis ---------------------------------------
// Source position of each output sample of a growing axis: CImg walks
// curr += (old-1)/(new-1) in double, clamped to old-1 (CImg.h:28445-28452);
// the walk is sequential, so one thread writes the table.
__global__ void k_resize_table(int old_n, int new_n, int *__restrict__ src, double *__restrict__ frac) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const double fx = new_n > 1 ? ((double)old_n - 1.0) / (double)(new_n - 1) : 0.0;
    double curr = 0.0;
    for (int x = 0; x < new_n; ++x) {
        const unsigned s = (unsigned)curr;
        frac[x] = curr - (double)s;
        src[x] = (int)s;
        const double nxt = curr + fx, lim = (double)old_n - 1.0;
        curr = (nxt < lim) ? nxt : lim;
    }
}

// mode 0: moving average (resize type 2): output t covers [t*old, (t+1)*old)
// and source s covers [s*new, (s+1)*new) of a common grid; the overlaps are
// accumulated in source order and divided by the old extent.  mode 1:
// Catmull-Rom in double from the table, clamped to the float range.
__global__ void k_resize_axis(const ResizeAxis ra, const float *__restrict__ in, float *__restrict__ out) {
    const long long total = (long long)ra.ox * ra.oy * ra.oz * ra.nc;
    const long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (id >= total) return;
    long long rem = id;
    int o[3];
    o[0] = (int)(rem % ra.ox);
    rem /= ra.ox;
    o[1] = (int)(rem % ra.oy);
    rem /= ra.oy;
    o[2] = (int)(rem % ra.oz);
    const int ch = (int)(rem / ra.oz);
    const long long st[3] = {1, ra.ix, (long long)ra.ix * ra.iy};
    const int t = o[ra.axis];
    o[ra.axis] = 0;
    const float *line = in + ch * (long long)ra.ix * ra.iy * ra.iz + o[0] * st[0] + o[1] * st[1] + o[2] * st[2];
    const long long ss = st[ra.axis];
    float res;
    if (ra.mode == 0) {
        const unsigned long long oldn = (unsigned)ra.old_n, nn = (unsigned)ra.new_n;
        const unsigned long long lo = (unsigned long long)t * oldn, hi = lo + oldn;
        float acc = 0.0f;
        for (unsigned long long s = lo / nn; s <= (hi - 1) / nn; ++s) {
            const unsigned long long a = s * nn > lo ? s * nn : lo;
            const unsigned long long b = (s + 1) * nn < hi ? (s + 1) * nn : hi;
            acc += __ldg(line + s * ss) * (float)(unsigned)(b - a);
        }
        res = acc / (float)(unsigned)oldn;
    } else {
        const int s = __ldg(ra.src + t);
        const double f = __ldg(ra.frac + t);
        const int m = ra.old_n;
        const double val1 = (double)__ldg(line + s * ss);
        const double val0 = s > 0 ? (double)__ldg(line + (s - 1) * ss) : val1;
        const double val2 = s <= m - 2 ? (double)__ldg(line + (s + 1) * ss) : val1;
        const double val3 = s < m - 2 ? (double)__ldg(line + (s + 2) * ss) : val2;
        const double val = val1 + 0.5f * (f * (-val0 + val2) + f * f * (2 * val0 - 5 * val1 + 4 * val2 - val3) +
                                          f * f * f * (-val0 + 3 * val1 - 3 * val2 + val3));
        res = (float)(val < -FLT_MAX ? -FLT_MAX : val > FLT_MAX ? FLT_MAX : val);
    }
    o[ra.axis] = t;
    out[ch * (long long)ra.ox * ra.oy * ra.oz + o[0] + (long long)o[1] * ra.ox + (long long)o[2] * ra.ox * ra.oy] = res;
}

// CImg::get_gradient("xyz", 0): 3 planes of central differences, Neumann.
__global__ void __launch_bounds__(128) k_gradient(const Dims d, const float *__restrict__ img, float *__restrict__ g) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= d.x) return;
    const long long sy = d.x, sz = (long long)d.x * d.y, n = sz * d.z;
    const long long p = i + j * sy + k * sz;
    const long long xm = i > 0 ? p - 1 : p, xp = i < d.x - 1 ? p + 1 : p;
    const long long ym = j > 0 ? p - sy : p, yp = j < d.y - 1 ? p + sy : p;
    const long long zm = k > 0 ? p - sz : p, zp = k < d.z - 1 ? p + sz : p;
    g[p] = (__ldg(img + xp) - __ldg(img + xm)) / 2;
    g[n + p] = (__ldg(img + yp) - __ldg(img + ym)) / 2;
    g[2 * n + p] = (__ldg(img + zp) - __ldg(img + zm)) / 2;
}

// The dual inside the ROI to the caller's planes (the write-back of
// optical_flow.h:503-533).
__global__ void __launch_bounds__(128) k_flow_unpack(const Dims d, const FlowRoi roi, const float *__restrict__ y,
                                                     float *__restrict__ Y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= d.x || !in_roi(roi, d, i, j, k)) return;
    const unsigned n = d.x * d.y * d.z, p = i + j * d.x + k * d.x * d.y;
    const Dual q = load_dual(y, n, p);
#pragma unroll
    for (int c = 0; c < 10; ++c) Y[(size_t)c * n + p] = q.y[c];
}

inline dim3 vox_grid(const int *d, int zmul = 1) {
    return dim3((unsigned)((d[0] + 127) / 128), (unsigned)d[1], (unsigned)(d[2] * zmul));
}

}  // namespace

cudaError_t launch_warp_box(const int *dim, const float *box, const float *vel, const float *src, int nc, float dt,
                            float *out, cudaStream_t s) {
    const dim3 grid((dim[0] + BOX_X - 1) / BOX_X, (dim[1] + BOX_Y - 1) / BOX_Y, dim[2]);
    const auto kernel = (long long)dim[0] * dim[1] * dim[2] < (1LL << 31) ? k_warp_box<int> : k_warp_box<long long>;
    kernel<<<grid, dim3(BOX_X, BOX_Y), 0, s>>>(Dims{dim[0], dim[1], dim[2]}, box[0], box[1], box[2], vel, src, nc, dt,
                                               out, -0.0f);
    return cudaGetLastError();
}

cudaError_t launch_flow_pack(long long n, const float *Y, const float *V, float *y, float4 *v0, float4 *v1, float4 *v2,
                             cudaStream_t s) {
    k_flow_pack<<<(unsigned)((n + 255) / 256), 256, 0, s>>>((unsigned)n, Y, V, y, v0, v1, v2);
    return cudaGetLastError();
}

cudaError_t launch_flow_setup(const int *d, const FlowRoi &roi, const float *i2w, const float *i1, const float *V,
                              float4 *u, float4 *steps, float *k4prev, cudaStream_t s) {
    k_flow_setup<<<vox_grid(d), 128, 0, s>>>(Dims{d[0], d[1], d[2]}, roi, i2w, i1, V, u, steps, k4prev);
    return cudaGetLastError();
}

cudaError_t launch_flow_primal(const int *d, const FlowRoi &roi, const float *y, const float4 *u, const float4 *steps,
                               const float4 *v_in, float4 *v_out, float *kty, int flags, double *resid,
                               const int *done, cudaStream_t s) {
    return launch_chained(k_flow_primal, vox_grid(d), 128, s, Dims{d[0], d[1], d[2]}, roi, y, u, steps, v_in, v_out,
                          kty, flags, resid, done);
}

namespace {
DualPar dual_par(float sigma1, float hf, float lambda, int huber) {
    // lam2_lo = lambda^2 (1 - 2^-20) rounded down: s < lam2_lo gives sqrt(s) < lambda (1 - 2^-21), whose float
    // rounding stays below lambda, so sqrt(s)/lambda rounds to at most 1.
    const double l2 = (double)lambda * (double)lambda * (1.0 - 1.0 / 1048576.0);
    float lam2_lo = (float)l2;
    if ((double)lam2_lo > l2) lam2_lo = std::nextafter(lam2_lo, 0.0f);
    return DualPar{sigma1, hf, lambda, lam2_lo, huber};
}
}  // namespace

cudaError_t launch_flow_dual(const int *d, const float4 *v, const float4 *v_old, const float4 *u, const float4 *steps,
                             const float *k4prev, float *y, float sigma1, float hf, float lambda, int huber, int flags,
                             double *resid, const int *done, cudaStream_t s) {
    return launch_chained(k_flow_dual, vox_grid(d), 128, s, Dims{d[0], d[1], d[2]}, v, v_old, u, steps, k4prev, y,
                          dual_par(sigma1, hf, lambda, huber), flags, resid, done);
}

// Whether the steps between residual checks run fused.  The two kernels update
// the dual in place, so they hold 120 bytes per voxel where k_flow_step holds
// 160: for the sizes in between, the two kernels' fields still stay in the L2
// (126 MB) from one iteration to the next and the fused kernel's don't.  Two
// kernels / fused, us per iteration: 72^3 (160 n = 0.45 of the L2) 14.7 / 13.6,
// 80^3 (0.62) 17.7 / 16.5, 90^3 (0.88) 23.1 / 25.8, 96^3 (1.07) 28.0 / 32.7, 97 x 96
// x 99 (1.11) 30.9 / 34.1, 104^3 (1.36) 40.5 / 41.5, 110^3 (1.60) 48.2 / 45.6,
// 124^3 (2.30) 67.0 / 60.4, 256^3 569 / 528.
bool flow_fuses(long long voxels) {
    int dev = 0, l2 = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess) cudaGetLastError();
    return voxels * 160 < l2 * 3LL / 4 || voxels * 160 > l2 * 3LL / 2;
}

cudaError_t launch_flow_step(const int *d, const FlowRoi &roi, const float *y_in, float *y_out, const float4 *v,
                             const float4 *v_old, float4 *v_next, const float4 *u, const float4 *steps,
                             const float *k4prev, float *kty, float sigma1, float hf, float lambda, int huber,
                             int flags, const int *done, cudaStream_t s) {
    const int gx = (d[0] + 30) / 31, gy = (d[1] + STEP_Y - 1) / STEP_Y;
    // Runs along z: the count whose rounds of resident blocks (four per SM) walk
    // the fewest planes, each run with about one and a half on top (the duals
    // formed again below it, and its first loads).
    const int resident = 4 * sm_count();
    int planes = d[2];
    long long best = -1;
    for (int runs = 1; runs <= std::max(1, d[2] / 3); ++runs) {
        const int pl = (d[2] + runs - 1) / runs;
        const long long blocks = (long long)gx * gy * ((d[2] + pl - 1) / pl);
        const long long cost = (blocks + resident - 1) / resident * (2 * pl + 3);
        if (best < 0 || cost < best) best = cost, planes = pl;
    }
    return launch_chained(k_flow_step, dim3(gx, gy, (d[2] + planes - 1) / planes), dim3(32, STEP_Y + 1), s,
                          Dims{d[0], d[1], d[2]}, roi, y_in, y_out, v, v_old, v_next, u, steps, k4prev, kty,
                          dual_par(sigma1, hf, lambda, huber), flags, planes, done);
}

cudaError_t launch_flow_settle(long long n, const int *iters, const float4 *v_1, const float4 *v_2, float4 *v_0,
                               float *V, cudaStream_t s) {
    k_flow_settle<<<(unsigned)((n + 255) / 256), 256, 0, s>>>((unsigned)n, iters, v_1, v_2, v_0, V);
    return cudaGetLastError();
}

cudaError_t launch_flow_check(double *resid, long long n, float tol, int it, int is_resid, int is_last, int *done,
                              int *iters, float *err, cudaStream_t s) {
    k_flow_check<<<1, 1, 0, s>>>(resid, n, tol, it, is_resid, is_last, done, iters, err);
    return cudaGetLastError();
}

cudaError_t launch_flow_reset(int *done, double *resid, int *iters, float *err, cudaStream_t s) {
    k_flow_reset<<<1, 1, 0, s>>>(done, resid, iters, err);
    return cudaGetLastError();
}

cudaError_t launch_deriche(const int *d, int nc, int axis, const DericheCoef &c, float *img, float *tmp,
                           cudaStream_t s) {
    const long long per_ch =
        axis == 0 ? (long long)d[1] * d[2] : axis == 1 ? (long long)d[0] * d[2] : (long long)d[0] * d[1];
    const long long lines = per_ch * nc;
    k_deriche_line<<<(unsigned)((lines + 127) / 128), 128, 0, s>>>(Dims{d[0], d[1], d[2]}, nc, axis, c, img, tmp);
    return cudaGetLastError();
}

cudaError_t launch_resize_table(int old_n, int new_n, int *src, double *frac, cudaStream_t s) {
    k_resize_table<<<1, 1, 0, s>>>(old_n, new_n, src, frac);
    return cudaGetLastError();
}

cudaError_t launch_resize_axis(const ResizeAxis &ra, const float *in, float *out, cudaStream_t s) {
    const long long total = (long long)ra.ox * ra.oy * ra.oz * ra.nc;
    k_resize_axis<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(ra, in, out);
    return cudaGetLastError();
}

cudaError_t launch_gradient(const int *d, const float *img, float *g, cudaStream_t s) {
    k_gradient<<<vox_grid(d), 128, 0, s>>>(Dims{d[0], d[1], d[2]}, img, g);
    return cudaGetLastError();
}

cudaError_t launch_flow_unpack(const int *d, const FlowRoi &roi, const float *y, float *Y, cudaStream_t s) {
    k_flow_unpack<<<vox_grid(d), 128, 0, s>>>(Dims{d[0], d[1], d[2]}, roi, y, Y);
    return cudaGetLastError();
}

}  // namespace stt
