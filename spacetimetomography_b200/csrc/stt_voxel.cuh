// stt_voxel.cuh -- device helpers of the voxel-driven steps, shared by the
// per-view kernels (k_voxel.cu) and the persistent sweep (k_persist.cu): the
// ROI tests, the voxel-based backprojection of one voxel and of one column,
// and the ROI mask with the over-relaxation.
//
// Paths cited are relative to the reference project root (gmzang/SpaceTimeTomography);
// S/ = SpaceTimeTomography/.
#pragma once

#include <climits>

#include "stt_internal.cuh"

namespace stt {

// ROI box of the primal-dual loops (ST_Tomography.cpp:514, 565, 593).
__device__ __forceinline__ bool roi_out(int i, int j, int k, int nx, int ny, int nz, const int *cut) {
    return i < cut[0] || i > nx - cut[1] || j < cut[2] || j > ny - cut[3] || k < cut[4] ||
           k > nz - cut[5];
}

// ROI mask (ST_Tomography.cpp:303-329); note the literal 7 in the y test of :324.
__device__ __forceinline__ float roi_value(int i, int j, int k, int nx, int ny, int nz, const int *cut) {
    float r = 1.0f;
    if (((i < cut[6]) && (k < cut[7])) || ((i < cut[6]) && (k > (nz - cut[7])))) r = 0.0f;
    if (((i > (nx - cut[6])) && (k < cut[7])) || ((i > (nx - cut[6])) && (k > (nz - cut[7])))) r = 0.0f;
    if (((k < cut[6]) && (i < cut[7])) || ((k < cut[6]) && (i > (nx - cut[7])))) r = 0.0f;
    if (((k > (nz - cut[6])) && (i < cut[7])) || ((k > (nz - cut[6])) && (i > (nx - cut[7])))) r = 0.0f;
    if (i < cut[0] || i > nx - cut[1] || j < cut[2] || j > ny - 7 || k < cut[4] || k > nz - cut[5]) r = 0.0f;
    return r;
}

struct Cut8 {
    int c[8];
};

// End of a SART call (ST_Tomography.cpp:793-804) for voxel (i, j, k),
// optionally fused with the over-relaxation that follows it in the
// primal-dual loop (:586-604): vol *= roi; if xbar: xbar = 2*vol - xprev in
// the ROI box.  vol is read with a plain load (a launch may have written it).
template <typename T>
__device__ __forceinline__ void roi_apply_at(int i, int j, int k, int nx, int ny, int nz, const int *cut,
                                             const int *pdcut, T *vol, const T *xprev, T *xbar) {
    const size_t p = i + (size_t)j * nx + (size_t)k * nx * ny;
    const bool kept = roi_value(i, j, k, nx, ny, nz, cut) != 0.0f;
    const bool relax = xbar && !roi_out(i, j, k, nx, ny, nz, pdcut);
    if (kept && !relax) return;  // times one: the voxel stays as it is
    float v = ld_stored(vol + p);
    if (!kept) {
        v *= 0.0f;  // (the reference's product: a NaN stays one, a negative voxel becomes -0)
        st_stored(vol + p, v);
    }
    if (relax) st_stored(xbar + p, 2.0f * v - ld_voxel(xprev + p));
}

// A load of an FP32 array: through the read-only path, or (RW) a plain load
// for an array that the running launch has written (the persistent sweep).
template <bool RW>
__device__ __forceinline__ float ld_f(const float *p) {
    if constexpr (RW) return *p;
    else return __ldg(p);
}

// Dual step of one frame at voxel (i, j, k) (ST_Tomography.cpp:504-534), fused:
//   whole volume:     ytp += sigma*(xf1 - xf);  ybc += sigma*(bw - xf)
//   interior & ROI:   ytv_c += sigma*(xf(p+e_c) - xf(p))*hf, clamp +-tv_w;
//                     ytp = ytp*tp_w/(tp_w + 2 sigma);  ybc clamp +-bc_w
// bw: the backward-warped X_bar[f+1] at the voxel.  T: the storage of X_bar
// (the duals are FP32).
template <typename T>
__device__ __forceinline__ void pd_dual_at(int i, int j, int k, int nx, int ny, int nz, float sigma, float tv_w,
                                           float tp_w, float bc_w, float hf, const int *cut, const T *xf,
                                           const T *xf1, float bw, float *ytv, float *ytp, float *ybc) {
    const size_t sy = nx, sz = (size_t)nx * ny, n = sz * nz;
    const size_t p = i + j * sy + k * sz;
    const float x0 = ld_voxel(xf + p);
    float tp = ytp[p] + sigma * (ld_voxel(xf1 + p) - x0);
    float bc = ybc[p] + sigma * (bw - x0);
    const bool inner = i >= 1 && i < nx - 1 && j >= 1 && j < ny - 1 && k >= 1 && k < nz - 1 &&
                       !roi_out(i, j, k, nx, ny, nz, cut);
    if (inner) {
        float y0 = ytv[p] + sigma * (ld_voxel(xf + p + 1) - x0) * hf;
        float y1 = ytv[p + n] + sigma * (ld_voxel(xf + p + sy) - x0) * hf;
        float y2 = ytv[p + 2 * n] + sigma * (ld_voxel(xf + p + sz) - x0) * hf;
        ytv[p] = rmax(-tv_w, rmin(tv_w, y0));
        ytv[p + n] = rmax(-tv_w, rmin(tv_w, y1));
        ytv[p + 2 * n] = rmax(-tv_w, rmin(tv_w, y2));
        tp = __fdiv_rn(tp * tp_w, tp_w + 2.0f * sigma);
        bc = rmax(-bc_w, rmin(bc_w, bc));
    }
    ytp[p] = tp;
    ybc[p] = bc;
}

// Primal step of one frame at voxel (i, j, k) (ST_Tomography.cpp:536-578),
// fused: xprev = vol; vol -= tau*(-ytp); vol -= tau*(-ybc) for the first
// frame, otherwise vol -= tau*(ytp_prev - ytp); vol -= tau*(fw - ybc); then
// on the interior ROI vol -= tau*(-div ytv) and clamp to [0, gmax].  fw: the
// forward-warped Y_bc[f-1] at the voxel.  T: the storage of vol and xprev
// (the duals are FP32).  RW: the duals were written by the same launch.
template <bool RW, typename T>
__device__ __forceinline__ void pd_primal_at(int i, int j, int k, int nx, int ny, int nz, float tau, float gmax,
                                             const int *cut, int first, const float *ytp_prev, const float *ytp,
                                             float fw, const float *ybc, const float *ytv, T *vol, T *xprev) {
    const size_t sy = nx, sz = (size_t)nx * ny, n = sz * nz;
    const size_t p = i + j * sy + k * sz;
    float v = ld_stored(vol + p);
    st_stored(xprev + p, v);
    if (first) {
        v = v - tau * (-ld_f<RW>(ytp + p));
        v = v - tau * (-ld_f<RW>(ybc + p));
    } else {
        v = v - tau * (ld_f<RW>(ytp_prev + p) - ld_f<RW>(ytp + p));
        v = v - tau * (fw - ld_f<RW>(ybc + p));
    }
    const bool inner = i >= 1 && i < nx - 1 && j >= 1 && j < ny - 1 && k >= 1 && k < nz - 1 &&
                       !roi_out(i, j, k, nx, ny, nz, cut);
    if (inner) {
        const float *y0 = ytv, *y1 = ytv + n, *y2 = ytv + 2 * n;
        float y = -(ld_f<RW>(y0 + p) - ld_f<RW>(y0 + p - 1) + ld_f<RW>(y1 + p) - ld_f<RW>(y1 + p - sy) +
                    ld_f<RW>(y2 + p) - ld_f<RW>(y2 + p - sz));
        v = v - tau * y;
        v = rmax(rmin(gmax, v), 0.0f);
    }
    st_stored(vol + p, v);
}

// Voxel-based backprojection (ST_Tomography.cpp:690-730): project the voxel
// centre, Catmull-Rom 4x4 gather of the correction image (y first, then x),
// vol += alpha*val, clamp to [0, gmax]; voxels projecting outside
// [2, W-2) x [2, H-2) are untouched.  Every product and sum is rounded on its
// own (explicit intrinsics), so the per-voxel and the column forms below give
// the same bits whichever way their taps are fetched.

// Camera coordinate r of voxel (fx, fy, fz): A[r]*(x, y, z) + b[r].
__device__ __forceinline__ float bp_cam(const ViewRec &v, int r, float fx, float fy, float fz) {
    return __fadd_rn(__fmaf_rn(v.A[3 * r + 2], fz, __fmaf_rn(v.A[3 * r + 1], fy, __fmul_rn(v.A[3 * r], fx))), v.b[r]);
}

// One detector axis of a voxel: the coordinate u = c + cam sdd/(ds depth), its
// 4-tap window's second tap p and the fraction d, and whether the voxel is
// used at all (2 <= u < n - 2, the reference's cutoff).  sdd/(ds depth) is
// formed once per depth (bp_scale), so a coordinate is one multiply-add; the
// cutoff, which is a jump, is decided within BP_NEAR pixels of a border by the
// coordinate as ST_Tomography.cpp:698-709 forms it, c + (cam/depth) sdd/ds, in
// its operation order.  u does not fall as cam grows.
constexpr float BP_NEAR = 0.0625f;

__device__ __forceinline__ float bp_scale(const GeomDev &g, float ndepth) { return __fdiv_rn(g.sdd_ds, ndepth); }
__device__ __forceinline__ float bp_coord(float c, float cam, float scale) { return __fmaf_rn(cam, scale, c); }
__device__ __forceinline__ bool bp_inside(const GeomDev &g, float u, float c, float cam, float ndepth, int n) {
    const float lo = 2.0f, hi = (float)(n - 2);
    if (u >= lo + BP_NEAR && u < hi - BP_NEAR) return true;
    if (!(u >= lo - BP_NEAR && u < hi + BP_NEAR)) return false;
    const float e = __fmaf_rn(__fdiv_rn(cam, ndepth), g.sdd_ds, c);
    return e >= lo && e < hi;
}
__device__ __forceinline__ int bp_tap(float u, int n) { return min(max((int)u, 2), n - 3); }

// Catmull-Rom weights of taps (-1, 0, +1, +2) at fraction d, in Horner form.
__device__ __forceinline__ void bp_weights(float d, float w[4]) {
    w[0] = __fmul_rn(d, __fmaf_rn(d, __fmaf_rn(-0.5f, d, 1.0f), -0.5f));
    w[1] = __fmaf_rn(__fmul_rn(d, d), __fmaf_rn(1.5f, d, -2.5f), 1.0f);
    w[2] = __fmul_rn(d, __fmaf_rn(d, __fmaf_rn(-1.5f, d, 2.0f), 0.5f));
    w[3] = __fmul_rn(__fmul_rn(d, d), __fmaf_rn(0.5f, d, -0.5f));
}

// The window's sum, rows first: bp_row is one detector row's four taps
// (columns px-1 .. px+2) under the x weights, bp_sum the four rows' sums
// under the y weights.  A row's sum depends on the row and the column's x
// weights only, so a column of voxels shares it (bp_column keeps a window of
// four, k_bp_voxel_cols a table).
__device__ __forceinline__ float bp_row(const float tap[4], const float wx[4]) {
    return __fmaf_rn(wx[3], tap[3], __fmaf_rn(wx[2], tap[2], __fmaf_rn(wx[1], tap[1], __fmul_rn(wx[0], tap[0]))));
}
__device__ __forceinline__ float bp_sum(const float row[4], const float wy[4]) {
    return __fmaf_rn(wy[3], row[3], __fmaf_rn(wy[2], row[2], __fmaf_rn(wy[1], row[1], __fmul_rn(wy[0], row[0]))));
}

// The updated voxel: v + alpha*val clamped to [0, gmax] as the reference's
// macros clamp (a NaN becomes 0).  top = bp_top(gmax), so that two plain
// minimum / maximum operations do it.
__device__ __forceinline__ float bp_top(float gmax) { return gmax != gmax ? INFINITY : fmaxf(gmax, 0.0f); }
__device__ __forceinline__ float bp_value(float v, float alpha, float val, float top) {
    return fminf(top, fmaxf(__fmaf_rn(alpha, val, v), 0.0f));
}
// T: the volume's storage (float, or BF16 bits widened to FP32 and rounded
// back to nearest even on store).
template <typename T>
__device__ __forceinline__ void bp_update(T *__restrict__ vol, size_t o, float alpha, float val, float top) {
    st_stored(vol + o, bp_value(ld_stored(vol + o), alpha, val, top));
}

// Fetchers of one correction row, pyr, at columns px-1 .. px+2.
// From the correction array through the read-only path (written by an
// earlier launch).
struct BpRowsLdg {
    const float *corr;
    int W;
    __device__ __forceinline__ void operator()(int px, int pyr, float r[4]) const {
        const float *c = corr + (size_t)pyr * W + (px - 1);
#pragma unroll
        for (int a = 0; a < 4; ++a) r[a] = __ldca(c + a);
    }
};
// From the correction array with plain loads (written by the same launch).
struct BpRowsLoad {
    const float *corr;
    int W;
    __device__ __forceinline__ void operator()(int px, int pyr, float r[4]) const {
        const float *c = corr + (size_t)pyr * W + (px - 1);
#pragma unroll
        for (int a = 0; a < 4; ++a) r[a] = ld_stored(c + a);
    }
};

// One voxel, everything computed for it alone.
template <typename Rows, typename T>
__device__ __forceinline__ void bp_voxel_at(const GeomDev &g, const ViewRec &v, const Rows &rows, T *__restrict__ vol,
                                            int x, int y, int z, float alpha, float gmax) {
    const float fx = (float)x, fy = (float)y, fz = (float)z;
    const float ndepth = -bp_cam(v, 2, fx, fy, fz);
    const float scale = bp_scale(g, ndepth), camx = bp_cam(v, 0, fx, fy, fz), camy = bp_cam(v, 1, fx, fy, fz);
    const float upx = bp_coord(g.cx, camx, scale), upy = bp_coord(g.cy, camy, scale);
    if (!bp_inside(g, upx, g.cx, camx, ndepth, g.W) || !bp_inside(g, upy, g.cy, camy, ndepth, g.H)) return;
    const int px = bp_tap(upx, g.W), py = bp_tap(upy, g.H);
    float wx[4], wy[4], s[4];
    bp_weights(upx - (float)px, wx);
    bp_weights(upy - (float)py, wy);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        float r[4];
        rows(px, py - 1 + b, r);
        s[b] = bp_row(r, wx);
    }
    bp_update(vol, x + (size_t)y * g.nx + (size_t)z * g.nx * g.ny, alpha, bp_sum(s, wy), bp_top(gmax));
}

// The column walk: voxels (x, y0 .. y0+K-1, z).  For a view whose matrix has
// A[1] == A[7] == 0 (every rotation about y) the voxel's detector column and
// depth do not depend on y: they are computed once (the y term of their sums
// is an exact zero, so the values are the per-voxel ones).  The detector row
// moves by about sdd/sid per voxel, and the window's four row sums are kept in
// registers: a step of 0 to 3 rows reuses the overlap and forms the new ones.
// Other views take the per-voxel form.
template <int K, typename Rows, typename T>
__device__ __forceinline__ void bp_column(const GeomDev &g, const ViewRec &v, const Rows &rows, T *__restrict__ vol,
                                          int x, int y0, int z, float alpha, float gmax) {
    const int y1 = min(y0 + K, g.ny);
    if (!(v.A[1] == 0.0f && v.A[7] == 0.0f)) {
        for (int y = y0; y < y1; ++y) bp_voxel_at(g, v, rows, vol, x, y, z, alpha, gmax);
        return;
    }
    const float fx = (float)x, fz = (float)z;
    const float ndepth = -bp_cam(v, 2, fx, (float)y0, fz);
    const float scale = bp_scale(g, ndepth), camx = bp_cam(v, 0, fx, (float)y0, fz), upx = bp_coord(g.cx, camx, scale);
    if (!bp_inside(g, upx, g.cx, camx, ndepth, g.W)) return;
    const int px = bp_tap(upx, g.W);
    float wx[4];
    bp_weights(upx - (float)px, wx);
    float s[4];  // s[b]: the sum of row pyc-1+b
    int pyc = INT_MIN / 2;
    for (int y = y0; y < y1; ++y) {
        const float camy = bp_cam(v, 1, fx, (float)y, fz), upy = bp_coord(g.cy, camy, scale);
        if (!bp_inside(g, upy, g.cy, camy, ndepth, g.H)) continue;
        const int py = bp_tap(upy, g.H);
        float wy[4];
        bp_weights(upy - (float)py, wy);
        int have = 0;  // rows kept
        if (py >= pyc && py <= pyc + 3) {
            have = 4 - (py - pyc);
            for (int k = pyc; k < py; ++k) s[0] = s[1], s[1] = s[2], s[2] = s[3];
        }
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (b >= have) {
                float r[4];
                rows(px, py - 1 + b, r);
                s[b] = bp_row(r, wx);
            }
        pyc = py;
        bp_update(vol, x + (size_t)y * g.nx + (size_t)z * g.nx * g.ny, alpha, bp_sum(s, wy), bp_top(gmax));
    }
}

}  // namespace stt
