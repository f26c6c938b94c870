// k_voxel.cu -- voxel-driven kernels: the voxel-based (gather) backprojector,
// the primal-dual dual/primal/over-relaxation steps and the ROI mask.
//
// All of these stream the volume once in x-fastest order: one thread per
// voxel along x, blocks of 128 threads, grid (ceil(nx/128), ny, nz), so every
// warp reads and writes 128 contiguous bytes per array.  The stencil
// neighbours (x+-1, y+-1, z+-1) come from L1/L2.
#include "stt_internal.cuh"
#include "stt_kernels.h"
#include "stt_voxel.cuh"

namespace stt {

namespace {

// Voxel-based backprojection, columns of K voxels up y; a block has 32 (x) by
// 4 (z) of them.  The detector column, the depth and the x weights are the
// column's; the detector rows its voxels' windows cover are one run of about
// K sdd/sid + 4.  Phase 1 forms the x-weighted sum of every row of every
// column's run into a table in shared memory (4 loads each, none waiting for
// another); phase 2 combines 4 row sums per voxel, four voxels' loads at a
// time and one group ahead.  A warp is 8 x 4 columns in phase 1, whose rows and
// taps lie close together on the detector whatever the view, and 32 x 1 in
// phase 2, whose voxels are consecutive.
// A column whose rows do not fit in the table (a magnification above
// (BP_ROWS - 5) / (K - 1) rows per voxel) takes the walk (bp_column).
//
// Bound by L1 (tags and data of the row loads: 80 % of its peak) and issue
// (62 %).  The form before walked the voxels up y and fetched each one's two new
// rows with two tld4 of a texture copy of the correction, which ran at the
// texture unit's rate.  Per view, mean of 12 views (that form -> this one, us):
// 192^3 / 256^2 52.1 -> 28.1, 256^3 / 512^2 92.0 -> 68.6, 512^3 / 1024^2
// 718 (626 with an L2 prefetch) -> 480.  Measured and not kept: warps of 32 x 1
// columns in both phases (90-degree views 80 us at 256^3: their lanes' rows
// differ), of 16 x 2 (69) and 8 x 4 (78, the volume in 32-byte pieces); 48
// registers and 10 blocks (72); all K voxels loaded first (128 registers: 100).
constexpr int BP_ROWS = 40, BP_G = 4;
constexpr int BP_PITCH = 40;  // table columns of one z: 8 banks on from the last, so neither phase's warps conflict

// One column of a rotation about y: whether any voxel of [y0, y1) may be
// updated, and the run of rows (u does not fall with y: A[4] > 0).
struct BpCol {
    float ndepth, scale, ulo, uhi;
    int r0, nr;
    bool live;
};
__device__ __forceinline__ BpCol bp_col(const GeomDev &g, const ViewRec &v, float fx, float fz, int y0, int y1) {
    BpCol c;
    c.ndepth = -bp_cam(v, 2, fx, (float)y0, fz);
    c.scale = bp_scale(g, c.ndepth);
    c.ulo = bp_coord(g.cy, bp_cam(v, 1, fx, (float)y0, fz), c.scale);
    c.uhi = bp_coord(g.cy, bp_cam(v, 1, fx, (float)(y1 - 1), fz), c.scale);
    c.r0 = bp_tap(c.ulo, g.H) - 1;
    c.nr = bp_tap(c.uhi, g.H) + 3 - c.r0;
    const float camx = bp_cam(v, 0, fx, (float)y0, fz);
    c.live = c.uhi >= 2.0f - BP_NEAR && c.ulo < (float)(g.H - 2) + BP_NEAR &&
             bp_inside(g, bp_coord(g.cx, camx, c.scale), g.cx, camx, c.ndepth, g.W);
    return c;
}

// MIR: every voxel written goes to `mirror` (slices mpitch elements apart) too.
template <int K, int OCC, typename T, bool MIR>
__global__ void __launch_bounds__(128, OCC) k_bp_voxel_cols(const GeomDev g, const ViewRec *__restrict__ views,
                                                            const ViewSel sel, const float *__restrict__ corr,
                                                            T *__restrict__ vol, float alpha, float gmax,
                                                            T *__restrict__ mirror, size_t mpitch) {
    __shared__ float table[BP_ROWS * 4 * BP_PITCH];
    constexpr int RS = 4 * BP_PITCH;  // one row of every column
    cudaGridDependencySynchronize();  // (a chained launch)
    int local;
    const ViewRec &v = views[sel_view(sel, local)];
    const int y0 = blockIdx.y * K, y1 = min(y0 + K, g.ny);
    const bool rot_y = v.A[1] == 0.0f && v.A[7] == 0.0f;
    if (rot_y) {
        const int xl = (threadIdx.x >> 5) * 8 + (threadIdx.x & 7), zl = (threadIdx.x >> 3) & 3;
        const int x = blockIdx.x * 32 + xl, z = blockIdx.z * 4 + zl;
        const float fx = (float)x, fz = (float)z;
        const BpCol c = bp_col(g, v, fx, fz, y0, y1);
        if (x < g.nx && z < g.nz && c.live && c.nr <= BP_ROWS) {
            const float upx = bp_coord(g.cx, bp_cam(v, 0, fx, (float)y0, fz), c.scale);
            const int px = bp_tap(upx, g.W);
            float wx[4];
            bp_weights(upx - (float)px, wx);
            float *row = table + zl * BP_PITCH + xl;
            const float *d = corr + (size_t)c.r0 * g.W + (px - 1);  // (a detector may have more than 2^32 pixels)
#pragma unroll 4
            for (int i = 0; i < c.nr; ++i, d += g.W) {
                const float t[4] = {__ldca(d), __ldca(d + 1), __ldca(d + 2), __ldca(d + 3)};
                row[RS * i] = bp_row(t, wx);
            }
        }
    }
    __syncthreads();
    const int xl = threadIdx.x & 31, zl = threadIdx.x >> 5;
    const int x = blockIdx.x * 32 + xl, z = blockIdx.z * 4 + zl;
    if (x >= g.nx || z >= g.nz) return;
    const float fx = (float)x, fz = (float)z;
    const BpCol c = bp_col(g, v, fx, fz, y0, y1);
    T *col = vol + x + (size_t)y0 * g.nx + (size_t)z * g.nx * g.ny;
    T *mcol = MIR ? mirror + x + (size_t)y0 * g.nx + z * mpitch : nullptr;
    if (!rot_y || (c.live && c.nr > BP_ROWS)) {
        bp_column<K>(g, v, BpRowsLdg{corr, g.W}, vol, x, y0, z, alpha, gmax);
        if (MIR)
            for (int y = y0; y < y1; ++y, col += g.nx, mcol += g.nx) *mcol = *col;
        return;
    }
    if (!c.live) return;
    const float *row = table + zl * BP_PITCH + xl - RS * (c.r0 + 1);
    const float top = bp_top(gmax);
    if (y1 - y0 == K && c.ulo >= 2.0f + BP_NEAR && c.uhi < (float)(g.H - 2) - BP_NEAR) {  // every voxel is updated
        float vox[BP_G];
#pragma unroll
        for (int q = 0; q < BP_G; ++q) vox[q] = ld_stored(col + q * g.nx);
#pragma unroll 1
        for (int k = 0; k < K; k += BP_G) {
            float next[BP_G];
#pragma unroll
            for (int q = 0; q < BP_G; ++q)
                if (k + BP_G < K) next[q] = ld_stored(col + (BP_G + q) * g.nx);
#pragma unroll
            for (int q = 0; q < BP_G; ++q) {
                const float upy = bp_coord(g.cy, bp_cam(v, 1, fx, (float)(y0 + k + q), fz), c.scale);
                const int py = (int)upy;  // (inside: bp_tap leaves it)
                float wy[4];
                bp_weights(upy - (float)py, wy);
                const float *w = row + RS * py;
                const float s[4] = {w[0], w[RS], w[2 * RS], w[3 * RS]};
                const float nv = bp_value(vox[q], alpha, bp_sum(s, wy), top);
                st_stored(col + q * g.nx, nv);
                if (MIR) st_stored(mcol + q * g.nx, nv);
            }
            col += BP_G * g.nx;
            if (MIR) mcol += BP_G * g.nx;
#pragma unroll
            for (int q = 0; q < BP_G; ++q) vox[q] = next[q];
        }
        return;
    }
    for (int y = y0; y < y1; ++y, col += g.nx, mcol += MIR ? g.nx : 0) {
        const float camy = bp_cam(v, 1, fx, (float)y, fz), upy = bp_coord(g.cy, camy, c.scale);
        if (!bp_inside(g, upy, g.cy, camy, c.ndepth, g.H)) continue;
        const int py = bp_tap(upy, g.H);
        float wy[4];
        bp_weights(upy - (float)py, wy);
        const float *w = row + RS * py;
        const float s[4] = {w[0], w[RS], w[2 * RS], w[3 * RS]};
        const float nv = bp_value(ld_stored(col), alpha, bp_sum(s, wy), top);
        st_stored(col, nv);
        if (MIR) st_stored(mcol, nv);
    }
}

// The dual and primal steps of one frame (pd_dual_at, pd_primal_at in
// stt_voxel.cuh), one thread per voxel.
template <typename T>
__global__ void __launch_bounds__(128) k_pd_dual(int nx, int ny, int nz, float sigma, float tv_w,
                                                 float tp_w, float bc_w, float hf, Cut8 cut,
                                                 const T *__restrict__ xf,
                                                 const T *__restrict__ xf1,
                                                 const float *__restrict__ bw, float *__restrict__ ytv,
                                                 float *__restrict__ ytp, float *__restrict__ ybc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= nx) return;
    const size_t p = i + (size_t)j * nx + (size_t)k * nx * ny;
    pd_dual_at(i, j, k, nx, ny, nz, sigma, tv_w, tp_w, bc_w, hf, cut.c, xf, xf1, __ldg(bw + p), ytv, ytp, ybc);
}

template <typename T>
__global__ void __launch_bounds__(128) k_pd_primal(int nx, int ny, int nz, float tau, float gmax,
                                                   Cut8 cut, int first,
                                                   const float *__restrict__ ytp_prev,
                                                   const float *__restrict__ ytp,
                                                   const float *__restrict__ fw,
                                                   const float *__restrict__ ybc,
                                                   const float *__restrict__ ytv,
                                                   T *__restrict__ vol, T *__restrict__ xprev) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= nx) return;
    const size_t p = i + (size_t)j * nx + (size_t)k * nx * ny;
    pd_primal_at<false>(i, j, k, nx, ny, nz, tau, gmax, cut.c, first, ytp_prev, ytp, first ? 0.0f : __ldg(fw + p),
                        ybc, ytv, vol, xprev);
}

// Over-relaxation (ST_Tomography.cpp:586-604): xbar = 2*vol - xprev in the ROI box.
template <typename T>
__global__ void __launch_bounds__(128) k_pd_extrapolate(int nx, int ny, int nz, Cut8 cut,
                                                        const T *__restrict__ vol,
                                                        const T *__restrict__ xprev,
                                                        T *__restrict__ xbar) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= nx || roi_out(i, j, k, nx, ny, nz, cut.c)) return;
    const size_t p = i + (size_t)j * nx + (size_t)k * nx * ny;
    st_stored(xbar + p, 2.0f * ld_voxel(vol + p) - ld_voxel(xprev + p));
}

// End of a SART call (ST_Tomography.cpp:793-804) optionally fused with the
// over-relaxation that follows it in the primal-dual loop (:586-604)
// (roi_apply_at).
// A thread takes ROI_Y rows: without the over-relaxation most voxels are
// inside and not touched, and a block per row of 128 of them is all launch.  The
// mask alone, every voxel read and written a row a block -> this, us: 512^3 550
// -> 169, 256^3 76.5 -> 39.7, 256^3 in BF16 77 -> 31.5; bound by the launched
// blocks and the masked rim's partial lines.
constexpr int ROI_Y = 8;
template <typename T>
__global__ void __launch_bounds__(128) k_roi_apply(int nx, int ny, int nz, Cut8 cut, Cut8 pdcut,
                                                   T *__restrict__ vol,
                                                   const T *__restrict__ xprev,
                                                   T *__restrict__ xbar) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nx) return;
    const int j0 = blockIdx.y * ROI_Y, j1 = min(j0 + ROI_Y, ny);
#pragma unroll 4
    for (int j = j0; j < j1; ++j)
        roi_apply_at(i, j, (int)blockIdx.z, nx, ny, nz, cut.c, pdcut.c, vol, xprev, xbar);
}

__global__ void __launch_bounds__(128) k_roi_mask(int nx, int ny, int nz, Cut8 cut, float *__restrict__ roi) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= nx) return;
    roi[i + (size_t)j * nx + (size_t)k * nx * ny] = roi_value(i, j, k, nx, ny, nz, cut.c);
}

// ---- FP64 helpers of the power iteration --------------------------------------
// out[0] += sum a*b (FP64 products and sums; one double atomic per block).
__global__ void __launch_bounds__(256) k_dot_f64(long long n, const float *__restrict__ a,
                                                 const float *__restrict__ b, double *__restrict__ out) {
    double s = 0.0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
        s += (double)__ldg(a + k) * (double)__ldg(b + k);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    __shared__ double part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
        atomicAdd(out, t);
    }
}

// x *= 1/sqrt(*norm2) (the factor formed in FP64); x = 0 when the norm is 0.
__global__ void __launch_bounds__(256) k_scale_inv_sqrt(long long n, float *__restrict__ x,
                                                        const double *__restrict__ norm2) {
    const double q = *norm2;
    const float f = q > 0.0 ? (float)(1.0 / sqrt(q)) : 0.0f;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
        x[k] *= f;
}

// Seeded start vector: uniform in [0.5, 1.5) from SplitMix64 of (seed, index).
__global__ void __launch_bounds__(256) k_fill_seeded(long long n, unsigned long long seed, float *__restrict__ x) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        unsigned long long z = seed + 0x9E3779B97F4A7C15ULL * (unsigned long long)(k + 1);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
        z ^= z >> 31;
        x[k] = 0.5f + (float)(z >> 40) * (1.0f / 16777216.0f);
    }
}

dim3 vox_grid(int nx, int ny, int nz) { return dim3((nx + 127) / 128, ny, nz); }

Cut8 to_cut(const int *c) {
    Cut8 r;
    for (int q = 0; q < 8; ++q) r.c[q] = c ? c[q] : 0;
    return r;
}

}  // namespace

cudaError_t launch_dot_f64(long long n, const float *a, const float *b, double *out, cudaStream_t s) {
    k_dot_f64<<<grid_stride_blocks(n, 256), 256, 0, s>>>(n, a, b, out);
    return cudaGetLastError();
}

cudaError_t launch_scale_inv_sqrt(long long n, float *x, const double *norm2, cudaStream_t s) {
    k_scale_inv_sqrt<<<grid_stride_blocks(n, 256), 256, 0, s>>>(n, x, norm2);
    return cudaGetLastError();
}

cudaError_t launch_fill_seeded(long long n, unsigned long long seed, float *x, cudaStream_t s) {
    k_fill_seeded<<<grid_stride_blocks(n, 256), 256, 0, s>>>(n, seed, x);
    return cudaGetLastError();
}

namespace {
template <int K, int OCC, typename T>
cudaError_t bp_cols(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr, T *vol, float alpha,
                    float gmax, cudaStream_t s, T *mirror) {
    // Chained to the projection that writes corr: 128 views of 128^2 at 128^3 3.46
    // -> 3.21 ms.  (The projection is not chained to this: it reads the volume
    // through the texture path.)
    const dim3 grid((g.nx + 31) / 32, (g.ny + K - 1) / K, (g.nz + 3) / 4);
    if (mirror)
        return launch_chained(k_bp_voxel_cols<K, OCC, T, true>, grid, 128, s, g, views, sel, corr, vol, alpha, gmax, mirror,
                              fp_mirror_pitch((size_t)g.nx * g.ny));
    return launch_chained(k_bp_voxel_cols<K, OCC, T, false>, grid, 128, s, g, views, sel, corr, vol, alpha, gmax, mirror,
                          (size_t)0);
}

template <typename T>
cudaError_t bp_voxel_any(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr, T *vol,
                         float alpha, float gmax, cudaStream_t s, int bp_variant, T *mirror) {
    switch (bp_variant) {
    case 1: return bp_cols<8, 8>(g, views, sel, corr, vol, alpha, gmax, s, mirror);
    case 2: return bp_cols<20, 8>(g, views, sel, corr, vol, alpha, gmax, s, mirror);
    case 3: return bp_cols<16, 6>(g, views, sel, corr, vol, alpha, gmax, s, mirror);
    case 4: return bp_cols<12, 8>(g, views, sel, corr, vol, alpha, gmax, s, mirror);
    default: break;
    }
    if (g.bp_len == 4) return bp_cols<4, 8>(g, views, sel, corr, vol, alpha, gmax, s, mirror);
    if (g.bp_len == 8) return bp_cols<8, 8>(g, views, sel, corr, vol, alpha, gmax, s, mirror);
    if (g.bp_len == 12) return bp_cols<12, 8>(g, views, sel, corr, vol, alpha, gmax, s, mirror);
    return bp_cols<16, 8>(g, views, sel, corr, vol, alpha, gmax, s, mirror);
}

template <typename T>
cudaError_t pd_dual_any(const int *d, const PdParams &p, const T *xf, const T *xf1, const float *bw, float *ytv,
                        float *ytp, float *ybc, cudaStream_t s) {
    k_pd_dual<T><<<vox_grid(d[0], d[1], d[2]), 128, 0, s>>>(d[0], d[1], d[2], p.sigma, p.tv_w, p.tp_w, p.bc_w, p.hf,
                                                            to_cut(p.cut), xf, xf1, bw, ytv, ytp, ybc);
    return cudaGetLastError();
}

template <typename T>
cudaError_t pd_primal_any(const int *d, const PdParams &p, int first, const float *ytp_prev, const float *ytp,
                          const float *fw, const float *ybc, const float *ytv, T *vol, T *xprev, cudaStream_t s) {
    k_pd_primal<T><<<vox_grid(d[0], d[1], d[2]), 128, 0, s>>>(d[0], d[1], d[2], p.tau, p.gmax, to_cut(p.cut), first,
                                                              ytp_prev, ytp, fw, ybc, ytv, vol, xprev);
    return cudaGetLastError();
}

template <typename T>
cudaError_t roi_apply_any(const int *d, const int *roi_cut, const int *pd_cut, T *vol, const T *xprev, T *xbar,
                          cudaStream_t s) {
    k_roi_apply<T><<<vox_grid(d[0], (d[1] + ROI_Y - 1) / ROI_Y, d[2]), 128, 0, s>>>(
        d[0], d[1], d[2], to_cut(roi_cut), to_cut(pd_cut), vol, xprev, xbar);
    return cudaGetLastError();
}

template <typename T>
cudaError_t pd_extrapolate_any(const int *d, const int *cut, const T *vol, const T *xprev, T *xbar, cudaStream_t s) {
    k_pd_extrapolate<T><<<vox_grid(d[0], d[1], d[2]), 128, 0, s>>>(d[0], d[1], d[2], to_cut(cut), vol, xprev, xbar);
    return cudaGetLastError();
}
}  // namespace

int bp_default_len(double rows, long long voxels) {
    // (K - 1) steps of `rows` between the first and the last voxel, their
    // windows' 4 rows, and one for where the run starts within a row
    for (int k : {16, 12, 8})
        if ((k - 1) * rows + 5.0 <= BP_ROWS) return k;
    // Past that some columns of 8 walk, which takes a larger volume to hide.  Columns of
    // 8 / 4, us, views at 0 / 30 / 90 degrees: 64^3 at 12 rows a voxel 10/12/13 -> 9/9/9,
    // 96^3 at 6 10/19/13 -> 11/15/15, 128^3 at 8 18/25/25 -> 19/22/19, 160^3 at 5.4
    // 38/49/41 -> 36/45/41, 256^3 at 6 122/149/129 -> 127/154/139.
    return voxels < (1LL << 23) && 3 * rows + 5.0 <= BP_ROWS ? 4 : 8;
}

const char *bp_variant_name(int v) {
    static const char *names[kBpVariants] = {"columns of 16, 12, 8 or 4 voxels by the magnification, 8 blocks per SM",
                                             "columns of 8 voxels, 8 blocks per SM",
                                             "columns of 20 voxels, 8 blocks per SM",
                                             "columns of 16 voxels, 6 blocks per SM",
                                             "columns of 12 voxels, 8 blocks per SM"};
    return v >= 0 && v < kBpVariants ? names[v] : "?";
}

cudaError_t launch_bp_voxel(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                            float *vol, float alpha, float gmax, cudaStream_t s, int bp_variant, float *mirror) {
    return bp_voxel_any(g, views, sel, corr, vol, alpha, gmax, s, bp_variant, mirror);
}

cudaError_t launch_bp_voxel(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                            unsigned short *vol, float alpha, float gmax, cudaStream_t s, int bp_variant,
                            unsigned short *mirror) {
    return bp_voxel_any(g, views, sel, corr, vol, alpha, gmax, s, bp_variant, mirror);
}

cudaError_t launch_pd_dual(const int *d, const PdParams &p, const float *xf, const float *xf1,
                           const float *bw, float *ytv, float *ytp, float *ybc, cudaStream_t s) {
    return pd_dual_any(d, p, xf, xf1, bw, ytv, ytp, ybc, s);
}

cudaError_t launch_pd_dual(const int *d, const PdParams &p, const unsigned short *xf, const unsigned short *xf1,
                           const float *bw, float *ytv, float *ytp, float *ybc, cudaStream_t s) {
    return pd_dual_any(d, p, xf, xf1, bw, ytv, ytp, ybc, s);
}

cudaError_t launch_pd_primal(const int *d, const PdParams &p, int first, const float *ytp_prev,
                             const float *ytp, const float *fw, const float *ybc, const float *ytv,
                             float *vol, float *xprev, cudaStream_t s) {
    return pd_primal_any(d, p, first, ytp_prev, ytp, fw, ybc, ytv, vol, xprev, s);
}

cudaError_t launch_pd_primal(const int *d, const PdParams &p, int first, const float *ytp_prev,
                             const float *ytp, const float *fw, const float *ybc, const float *ytv,
                             unsigned short *vol, unsigned short *xprev, cudaStream_t s) {
    return pd_primal_any(d, p, first, ytp_prev, ytp, fw, ybc, ytv, vol, xprev, s);
}

cudaError_t launch_pd_extrapolate(const int *d, const int *cut, const float *vol, const float *xprev,
                                  float *xbar, cudaStream_t s) {
    return pd_extrapolate_any(d, cut, vol, xprev, xbar, s);
}

cudaError_t launch_pd_extrapolate(const int *d, const int *cut, const unsigned short *vol,
                                  const unsigned short *xprev, unsigned short *xbar, cudaStream_t s) {
    return pd_extrapolate_any(d, cut, vol, xprev, xbar, s);
}

cudaError_t launch_roi_apply(const int *d, const int *roi_cut, const int *pd_cut, float *vol,
                             const float *xprev, float *xbar, cudaStream_t s) {
    return roi_apply_any(d, roi_cut, pd_cut, vol, xprev, xbar, s);
}

cudaError_t launch_roi_apply(const int *d, const int *roi_cut, const int *pd_cut, unsigned short *vol,
                             const unsigned short *xprev, unsigned short *xbar, cudaStream_t s) {
    return roi_apply_any(d, roi_cut, pd_cut, vol, xprev, xbar, s);
}

cudaError_t launch_roi_mask(const int *d, const int *cut, float *roi, cudaStream_t s) {
    k_roi_mask<<<vox_grid(d[0], d[1], d[2]), 128, 0, s>>>(d[0], d[1], d[2], to_cut(cut), roi);
    return cudaGetLastError();
}

}  // namespace stt
