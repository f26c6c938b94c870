// k_warp.cu -- semi-Lagrangian tricubic warp (S/ST_Tomo/warping.h:49-145) and
// its vector-Jacobian product.
//
// One thread per output voxel, x fastest.  Per voxel: the velocity at the
// cell centre (an exact grid read: the Catmull-Rom sampler interpolates, and
// the centre lands on a node), one clamped tricubic velocity sample at the
// half-traced point (3 channels sharing one 64-tap stencil) and one clamped
// tricubic sample of every source channel at the traced point.  Taps come from
// L1/L2 through the read-only path; the cell corners of the clamp are taps of
// the stencil, so a sample is at most 64 loads per channel.  The kernel is
// bound by L1 load wavefronts, not by HBM.
#include <climits>

#include "stt_internal.cuh"
#include "stt_kernels.h"
#include "stt_tma.cuh"
#include "warp_dev.cuh"

namespace stt {

namespace {

using namespace warpdev;

// Blocks of 32 x 4 voxels: a warp is one x-run of 32, so every tap load of a
// warp reads ~32 consecutive floats, and the block's four rows share most of
// their stencil rows in L1.  All offsets are 32-bit (the host bounds
// n * max(nc, 3) below 2^31).
constexpr int WARP_BX = 32, WARP_BY = 4;

// T: the source's storage (float, or BF16 bits widened exactly to FP32).
template <typename T, typename I>
__global__ void __launch_bounds__(WARP_BX *WARP_BY) k_warp(const Dim3i d, const float *__restrict__ vel,
                                                           const T *__restrict__ src, int nc, float dt,
                                                           float *__restrict__ out) {
    const int i = blockIdx.x * WARP_BX + threadIdx.x;
    const int j = blockIdx.y * WARP_BY + threadIdx.y, k = blockIdx.z;
    if (i >= d.x || j >= d.y) return;
    const size_t n = (size_t)d.x * d.y * d.z;
    Cell<I> s;
    trace_cell(d, vel, dt, i, j, k, s);
    const I o = i + (I)j * d.x + (I)k * d.x * d.y;
    for (int ch = 0; ch < nc; ++ch) {
        float v[1];
        sample_cell<1>(src + ch * n, 0, s, v);
        out[o + ch * n] = v[0];
    }
}

// Staged form: the three velocity planes around the block's half-traced
// points come into shared memory with one 4D TMA box, and the velocity sample
// (three quarters of the warp's taps) reads them there.  Each thread finds the
// first tap of its velocity stencil after the exact centre read; the block's
// minimum places the box (x rounded down to 16 bytes); a stencil that does not
// fit in the box (a rough flow, a copy that did not land within the bounded
// wait) reads global memory.  The taps and the arithmetic are those of k_warp,
// so the outputs are the same bits.  The source sample stays on the L1 path.
constexpr int VX = 40, VY = 10, VZ = 6;  // velocity box (x, y, z) per plane; VX*4 is a multiple of 16
constexpr int VBOX = VX * VY * VZ;
constexpr long long WARP_WAIT_CYCLES = 200000000LL;  // about 0.1 s

// Status word of the warps launched without one (stt_warp, stt_warp_box on
// their own): one per device, read and cleared by stt_warp_poll_status.
__device__ int g_warp_wait_status;

template <typename T>
__global__ void __launch_bounds__(WARP_BX *WARP_BY) k_warp_staged(const Dim3i d,
                                                                  const __grid_constant__ CUtensorMap vmap,
                                                                  const float *__restrict__ vel,
                                                                  const T *__restrict__ src, int nc, float dt,
                                                                  float *__restrict__ out, int *status) {
    __shared__ alignas(128) float vbox[3 * VBOX];
    __shared__ uint64_t bar;
    __shared__ int red[3 * WARP_BY];
    const int i = blockIdx.x * WARP_BX + threadIdx.x;
    const int j = blockIdx.y * WARP_BY + threadIdx.y, k = blockIdx.z;
    const bool live = i < d.x && j < d.y;
    const size_t n = (size_t)d.x * d.y * d.z;
    const float h = -dt;
    const float p[3] = {(float)i + 0.5f, (float)j + 0.5f, (float)k + 0.5f};
    float p2[3] = {0.0f, 0.0f, 0.0f}, g2[3] = {1.0f, 1.0f, 1.0f};
    int b0[3] = {INT_MAX, INT_MAX, INT_MAX};  // first tap of the velocity stencil
    if (live) {
        // cell centre (warping.h:25-29); the velocity there is an exact node read
        const int ci = min(max(i, 1), d.x - 2), cj = min(max(j, 1), d.y - 2), ck = min(max(k, 1), d.z - 2);
        const int c = ci + cj * d.x + ck * d.x * d.y;
        const float v1[3] = {__ldg(vel + c), __ldg(vel + n + c), __ldg(vel + 2 * n + c)};
        // trace (warping.h:100-114): p2 = p + h v(p); p0 = p2 - h v(p2); q = p2 + (p - p0)/2
#pragma unroll
        for (int a = 0; a < 3; ++a) p2[a] = __fadd_rn(p[a], __fmul_rn(h, v1[a]));
        g2[0] = to_grid(p2[0], d.x, nullptr);
        g2[1] = to_grid(p2[1], d.y, nullptr);
        g2[2] = to_grid(p2[2], d.z, nullptr);
#pragma unroll
        for (int a = 0; a < 3; ++a) b0[a] = (int)g2[a] - 1;
    }
    int m[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) m[a] = __reduce_min_sync(0xffffffffu, b0[a]);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) red[3 * threadIdx.y + a] = m[a];
    }
    const bool lead = threadIdx.x == 0 && threadIdx.y == 0;
    if (lead) {
        tma::mbar_init(&bar, 1);
        tma::fence_barrier_init();
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        m[a] = red[a];
#pragma unroll
        for (int w = 1; w < WARP_BY; ++w) m[a] = min(m[a], red[3 * w + a]);
    }
    const bool any = m[0] != INT_MAX;  // uniform: some voxel of the block is inside the volume
    const int ox = (m[0] >> 2) << 2, oy = m[1], oz = m[2];
    if (any && lead) {
        tma::mbar_arrive_expect_tx(&bar, 3u * VBOX * sizeof(float));
        tma::load_box_4d(vbox, &vmap, ox, oy, oz, 0, &bar);
    }
    bool staged = false;
    if (any) {
        staged = tma::mbar_wait(&bar, 0, WARP_WAIT_CYCLES);
        if (!staged) {
            // An error, reported through the status word.  The velocity sample
            // reads global memory instead (same bits); the box is not read, but
            // the block waits (bounded) once more so that it does not exit with
            // the copy still writing into its shared memory.
            atomicExch(status ? status : &g_warp_wait_status, STT_WAIT_TIMEOUT_FLAG);
            tma::mbar_wait(&bar, 0, WARP_WAIT_CYCLES);
        }
    }
    if (!live) return;
    Cell<int> s2;
    cell_setup(d, g2, s2);
    float v2[3];
    const unsigned lx = (unsigned)(b0[0] - ox), ly = (unsigned)(b0[1] - oy), lz = (unsigned)(b0[2] - oz);
    if (staged && lx <= VX - 4 && ly <= VY - 4 && lz <= VZ - 4) {
        Cell<int> sl = s2;  // the same weights and edge flags, box-local offsets
        sl.sy = VX;
        sl.sz = VX * VY;
        sl.x.lo = (int)lx;
        sl.y.lo = (int)ly * VX;
        sl.z.lo = (int)lz * VX * VY;
        sample_cell<3, true>(vbox, VBOX, sl, v2);
    } else {
        sample_cell<3>(vel, n, s2, v2);
    }
    float q[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float p0 = __fsub_rn(p2[a], __fmul_rn(h, v2[a]));
        q[a] = __fadd_rn(p2[a], __fmul_rn(0.5f, __fsub_rn(p[a], p0)));
    }
    const float gq[3] = {to_grid(q[0], d.x, nullptr), to_grid(q[1], d.y, nullptr), to_grid(q[2], d.z, nullptr)};
    Cell<int> s;
    cell_setup(d, gq, s);
    const int o = i + j * d.x + k * d.x * d.y;
    for (int ch = 0; ch < nc; ++ch) {
        float v[1];
        sample_cell<1>(src + ch * n, 0, s, v);
        out[o + ch * n] = v[0];
    }
}

// ---- VJP ---------------------------------------------------------------
// One axis of a sample's stencil: the taps x-1, x, x+1, x+2 counted from the
// first (the last one held at the image's edge, where its weight is 0), their
// weights and the weights' slopes.  An axis whose coordinate was clamped to
// [1, dim-2] has no slope.
struct AxisD {
    int lo, last;
    float w[4], dw[4];
};

__device__ __forceinline__ void axis_d(float p, int dim, AxisD &a) {
    bool clamped;
    const float g = to_grid(p, dim, &clamped);
    const int x = (int)g;
    const float d = g - (float)x, d2 = d * d;
    cr_weights(d, a.w);
    a.dw[0] = 0.5f * (-1.0f + 4.0f * d - 3.0f * d2);
    a.dw[1] = 0.5f * (-10.0f * d + 9.0f * d2);
    a.dw[2] = 0.5f * (1.0f + 8.0f * d - 9.0f * d2);
    a.dw[3] = 0.5f * (-2.0f * d + 3.0f * d2);
    if (!(d > 0.0f)) a.dw[1] = a.dw[2], a.dw[2] = 0.0f;  // (on a node CImg's tap x+1 is x; dw[1] is 0 there)
    if (clamped)
#pragma unroll
        for (int k = 0; k < 4; ++k) a.dw[k] = 0.0f;
    a.lo = x - 1;
    a.last = x + 2 < dim ? 3 : 2;
}

struct CellD {
    AxisD x, y, z;
    int at;  // the first tap
};

__device__ __forceinline__ void cell_d(const Dim3i d, const float p[3], CellD &c) {
    axis_d(p[0], d.x, c.x);
    axis_d(p[1], d.y, c.y);
    axis_d(p[2], d.z, c.z);
    c.at = c.x.lo + c.y.lo * d.x + c.z.lo * d.x * d.y;
}

// One clamped sample: its value, which branch the clamp took (corner: the
// voxel it took, or -1) and, where it did not, the value's spatial gradient.
struct SampleD {
    float value;
    int corner;
    float grad[3];
};

__device__ __forceinline__ void sample_d(const Dim3i d, const float *__restrict__ img, const CellD &s, SampleD &r) {
    // Separable sums in the forward sampler's order (x taps, then rows, then
    // planes): per row its value and x-slope, per plane its value and x- and
    // y-slopes, then the sample's value and gradient.
    const int sy = d.x, sz = d.x * d.y;
    float val = 0.0f, gx = 0.0f, gy = 0.0f, gz = 0.0f, corner[8];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        float pv = 0.0f, px = 0.0f, py = 0.0f;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float *row = img + (s.at + (b < 3 ? b : s.y.last) * sy + (c < 3 ? c : s.z.last) * sz);
            const float t0 = __ldg(row), t1 = __ldg(row + 1), t2 = __ldg(row + 2), t3 = __ldg(row + s.x.last);
            const float xv = __fmaf_rn(s.x.w[3], t3, __fmaf_rn(s.x.w[2], t2, __fmaf_rn(s.x.w[0], t0, __fmul_rn(s.x.w[1], t1))));
            const float xd = s.x.dw[0] * t0 + s.x.dw[1] * t1 + s.x.dw[2] * t2 + s.x.dw[3] * t3;
            pv = __fmaf_rn(s.y.w[b], xv, pv);
            px += s.y.w[b] * xd;
            py += s.y.dw[b] * xv;
            if ((b == 1 || b == 2) && (c == 1 || c == 2)) {
                corner[2 * (b - 1) + 4 * (c - 1)] = t1;
                corner[2 * (b - 1) + 4 * (c - 1) + 1] = t2;
            }
        }
        val = __fmaf_rn(s.z.w[c], pv, val);
        gx += s.z.w[c] * px;
        gy += s.z.w[c] * py;
        gz += s.z.dw[c] * pv;
    }
    constexpr int order[7] = {1, 3, 2, 4, 5, 7, 6};  // (of equal corners the first in the reference's order)
    int imn = 0, imx = 0;
    float mn = corner[0], mx = mn;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        const float v = corner[order[k]];
        if (v < mn) mn = v, imn = order[k];
        if (mx < v) mx = v, imx = order[k];
    }
    const bool above = val > mx, below = !above && val < mn, in = !above && !below;
    const int m = above ? imx : imn;
    const float inner = (val < mx) ? val : mx;
    r.value = (mn < inner) ? inner : mn;
    r.corner = in ? -1 : s.at + 1 + (m & 1) + (1 + (m >> 1 & 1)) * sy + (1 + (m >> 2)) * sz;
    r.grad[0] = in ? gx : 0.0f;
    r.grad[1] = in ? gy : 0.0f;
    r.grad[2] = in ? gz : 0.0f;
}

// Which neighbours in the warp have the same cell one voxel on: left: the lane
// below samples the cell at x-1, right: the lane above the one at x+1.
struct Links {
    bool left, right;
};

__device__ __forceinline__ Links links_of(const CellD &s, const SampleD &r, bool live) {
    const int lane = threadIdx.x & 31;
    const int key = live && r.corner < 0 ? s.at : INT_MIN;
    // (cells of a row of voxels: at is one more exactly where x is, and y and z are the same: x+1 <= dim-2)
    const int below = __shfl_up_sync(0xffffffffu, key, 1), above = __shfl_down_sync(0xffffffffu, key, 1);
    Links l;
    l.left = lane > 0 && key != INT_MIN && below == key - 1;
    l.right = lane < 31 && key != INT_MIN && above == key + 1;
    return l;
}

// Adds g times a sample's weights to bar.  Every lane of the warp calls this.
// Lanes are neighbours along x, and so mostly are their cells: of the four taps
// of a row, three fall on voxels that neighbouring lanes add to as well.  Those go
// to the neighbour by shuffle, and a lane adds its own voxel's sum; the taps past
// the ends of a run of linked lanes are added on their own, one per lane and
// instruction.  (An atomic instruction costs the SM 4.7 cycles however few of its
// lanes are live, 7.4 for 32 adjacent floats, 11 for 32 in four rows; four a row
// without the merge.)
__device__ __forceinline__ void scatter_sample(const Dim3i d, float *__restrict__ bar, const CellD &s, const SampleD &r,
                                               float g, bool live) {
    live = live && g != 0.0f;
    if (!__any_sync(0xffffffffu, live)) return;
    if (live && r.corner >= 0) atomicAdd(bar + r.corner, g);
    const Links l = links_of(s, r, live);
    const bool mine = live && r.corner < 0;
    const bool ends = !l.left || !l.right, alone = !l.left && !l.right;
    const int sy = d.x, sz = d.x * d.y;
    float wx[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) wx[a] = mine ? g * s.x.w[a] : 0.0f;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
        const float wz = c == 0 ? s.z.w[0] : c == 1 ? s.z.w[1] : c == 2 ? s.z.w[2] : s.z.w[3];
        const int plane = s.at + (c < 3 ? c : s.z.last) * sz;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float f = s.y.w[b] * wz;
            const float w0 = wx[0] * f, w1 = wx[1] * f, w2 = wx[2] * f, w3 = wx[3] * f;
            const float u3 = __shfl_up_sync(0xffffffffu, w3, 1);
            const float e2 = w2 + (l.left ? u3 : 0.0f);  // what lies at x+1: mine and the left neighbour's last
            const float u2 = __shfl_up_sync(0xffffffffu, e2, 1), d0 = __shfl_down_sync(0xffffffffu, w0, 1);
            const float e1 = w1 + (l.left ? u2 : 0.0f) + (l.right ? d0 : 0.0f);
            float *row = bar + (plane + (b < 3 ? b : s.y.last) * sy);
            if (e1 != 0.0f) atomicAdd(row + 1, e1);
            // what no neighbour takes: the first tap of a run, the last two of its end
            const float out = l.left ? w3 : w0;
            if (ends && out != 0.0f) atomicAdd(row + (l.left ? s.x.last : 0), out);
            if (!l.right && e2 != 0.0f) atomicAdd(row + 2, e2);
            if (alone && w3 != 0.0f) atomicAdd(row + s.x.last, w3);
        }
    }
}

// q = p + (h/2) v(p) + (h/2) v(p2), p2 = p + h v(p).  Reverse mode:
//   out_c = S(src_c, q)        -> src_bar, q_bar
//   q_bar -> v2_bar = (h/2) q_bar;  p2_bar = q_bar/2 + J_v(p2)^T v2_bar
//   v1_bar = (h/2) q_bar' ... folded: v1_bar = h * p2_bar (p2 = p + h v1)
// The centre read v(p) is an exact node value, so its adjoint is a single add.
// One pass over the velocity taps gives the trace and the gradients, which only
// the reverse step uses.  Per voxel 256 taps, and 64 row sums of 2 to 3 atomic
// instructions, which bound it.  us, every tap an atomic, the velocity sampled
// again for its gradients, rows of 128 voxels -> this: 60 x 50 x 55 121 -> 79,
// 112 x 128 x 96 629 -> 401 (motion of 8 voxels: 793 -> 512), 256^3 6281 -> 4062.
// Five blocks per SM (96 registers): four 414, three 481, six 416 at 112 x 128 x 96.
__global__ void __launch_bounds__(WARP_BX *WARP_BY, 5) k_warp_vjp(const Dim3i d, const float *__restrict__ vel,
                                                               const float *__restrict__ src, int nc, float dt,
                                                               const float *__restrict__ out_bar,
                                                               float *__restrict__ src_bar,
                                                               float *__restrict__ vel_bar) {
    const int i = blockIdx.x * WARP_BX + threadIdx.x;
    const int j = blockIdx.y * WARP_BY + threadIdx.y, k = blockIdx.z;
    const bool live = i < d.x && j < d.y;
    const int n = d.x * d.y * d.z;
    const float h = -dt;
    // cell centre (warping.h:25-29) and the velocity there (an exact node read)
    const float p[3] = {(float)i + 0.5f, (float)j + 0.5f, (float)k + 0.5f};
    const int ci = min(max(i, 1), d.x - 2), cj = min(max(j, 1), d.y - 2), ck = min(max(k, 1), d.z - 2);
    const int centre = ci + cj * d.x + ck * d.x * d.y;
    float p2[3], q[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) p2[a] = __fadd_rn(p[a], __fmul_rn(h, __ldg(vel + (size_t)a * n + centre)));
    CellD s2, sq;
    cell_d(d, p2, s2);
    SampleD v2[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        sample_d(d, vel + (size_t)a * n, s2, v2[a]);
        const float p0 = __fsub_rn(p2[a], __fmul_rn(h, v2[a].value));
        q[a] = __fadd_rn(p2[a], __fmul_rn(0.5f, __fsub_rn(p[a], p0)));
    }
    cell_d(d, q, sq);
    const size_t o = i + (size_t)j * d.x + (size_t)k * d.x * d.y;
    float qbar[3] = {0.0f, 0.0f, 0.0f};
    for (int c = 0; c < nc; ++c) {
        const float ob = live ? __ldg(out_bar + o + (size_t)c * n) : 0.0f;
        SampleD r;
        r.corner = -1;
        if (ob != 0.0f) {
            sample_d(d, src + (size_t)c * n, sq, r);
#pragma unroll
            for (int a = 0; a < 3; ++a) qbar[a] += ob * r.grad[a];
        }
        if (src_bar) scatter_sample(d, src_bar + (size_t)c * n, sq, r, ob, live);
    }
    if (!vel_bar) return;
    const bool moves = qbar[0] != 0.0f || qbar[1] != 0.0f || qbar[2] != 0.0f;
    float p2bar[3] = {0.5f * qbar[0], 0.5f * qbar[1], 0.5f * qbar[2]};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float v2bar = 0.5f * h * qbar[a];
        scatter_sample(d, vel_bar + (size_t)a * n, s2, v2[a], v2bar, moves);
#pragma unroll
        for (int e = 0; e < 3; ++e) p2bar[e] += v2bar * v2[a].grad[e];
    }
    if (!moves) return;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float g = h * p2bar[a];
        if (g != 0.0f) atomicAdd(vel_bar + (size_t)a * n + centre, g);
    }
}

}  // namespace

cudaError_t warp_poll_status(int *flag, cudaStream_t s) {
    *flag = 0;
    cudaError_t e = cudaMemcpyFromSymbolAsync(flag, g_warp_wait_status, sizeof(int), 0, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && *flag) {
        const int zero = 0;
        e = cudaMemcpyToSymbolAsync(g_warp_wait_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    return e;
}

namespace {
template <typename T>
cudaError_t warp_any(const int *dim, const float *vel, const T *src, int nc, float dt, float *out, cudaStream_t s,
                     int *status) {
    Dim3i d{dim[0], dim[1], dim[2]};
    const dim3 grid((d.x + WARP_BX - 1) / WARP_BX, (d.y + WARP_BY - 1) / WARP_BY, d.z), block(WARP_BX, WARP_BY);
    CUtensorMap vmap;
    const unsigned box[4] = {VX, VY, VZ, 3};
    if (needs_general(d))
        k_warp<T, long long><<<grid, block, 0, s>>>(d, vel, src, nc, dt, out);
    else if (encode_planes_map(&vmap, vel, d.x, d.y, d.z, 3, box))
        k_warp_staged<T><<<grid, block, 0, s>>>(d, vmap, vel, src, nc, dt, out, status);
    else
        k_warp<T, int><<<grid, block, 0, s>>>(d, vel, src, nc, dt, out);
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_warp(const int *dim, const float *vel, const float *src, int nc, float dt,
                        float *out, cudaStream_t s, int *status) {
    return warp_any(dim, vel, src, nc, dt, out, s, status);
}

cudaError_t launch_warp(const int *dim, const float *vel, const unsigned short *src, int nc, float dt,
                        float *out, cudaStream_t s, int *status) {
    return warp_any(dim, vel, src, nc, dt, out, s, status);
}

cudaError_t launch_warp_vjp(const int *dim, const float *vel, const float *src, int nc, float dt,
                            const float *out_bar, float *src_bar, float *vel_bar, cudaStream_t s) {
    Dim3i d{dim[0], dim[1], dim[2]};
    const dim3 grid((d.x + WARP_BX - 1) / WARP_BX, (d.y + WARP_BY - 1) / WARP_BY, d.z), block(WARP_BX, WARP_BY);
    k_warp_vjp<<<grid, block, 0, s>>>(d, vel, src, nc, dt, out_bar, src_bar, vel_bar);
    return cudaGetLastError();
}

}  // namespace stt
