// k_project.cu -- the forward projection, and the forward projection fused with
// the SART correction.
//
// One thread per detector pixel.  A 128-thread block covers 32x4 pixels: each
// warp is 32 consecutive detector columns of one row, so at every step its 32
// samples lie along the detector's u axis in the volume.  For views whose rays
// run mostly along z, u maps to the volume's x axis, which is contiguous in
// memory; for views whose rays run mostly along x, u maps to z and the load
// forms of the forward projector gather from a z-fastest transposed copy
// (ViewRec::layout), so either way a warp's gathers touch few cache lines.  The
// texture forms (two tld4 per sample) read the volume itself for every view.
// The volume is read through the read-only path (ld.global.nc); at the headline
// sizes (256^3 fp32 = 64 MiB) it stays resident in the 126 MB L2.
#include "stt_internal.cuh"
#include "stt_kernels.h"

namespace stt {

namespace {

__device__ __forceinline__ bool tile_pixel(const GeomDev &g, int &i, int &j) {
    i = blockIdx.x * 32 + (threadIdx.x & 31);
    j = blockIdx.y * 4 + (threadIdx.x >> 5);
    return i < g.W && j < g.H;
}

// The ray sum gathered from the z-fastest transposed copy for layout-1 views
// when one is given, else from the volume (fp_ray_sum_with).
template <int FAST, typename I, int G = FP_GROUP, bool PK = false, typename T>
__device__ __forceinline__ float fp_ray_sum_from(const GeomDev &g, const T *__restrict__ src, const Strides &st,
                                                 const Ray &r, int *count) {
    return fp_ray_sum_with<G, PK>(
        g, [=](int, const FpCell &c, float v[8]) { fp_corners<FAST, I>(src, st, c, v); }, r, count);
}

// The ray sum through the texture of FpTex.
template <int G = FP_GROUP, bool PK = false, typename T = float>
__device__ __forceinline__ float fp_ray_sum_tex(const GeomDev &g, const FpTex &tex, const Ray &r, int *count) {
    const unsigned long long t = tex.x;
    const int nx = g.nx;
    return fp_ray_sum_with<G, PK>(
        g, [=](int, const FpCell &c, float w[8]) { fp_corners_tex<T>(t, nx, c, w); }, r, count);
}

template <typename I, int G = FP_GROUP, bool PK = false, typename T>
__device__ __forceinline__ float fp_ray_sum(const GeomDev &g, const ViewRec &v, const T *__restrict__ vol,
                                            const T *__restrict__ vol_t, const Ray &r, int *count) {
    if (vol_t && v.layout == 1) return fp_ray_sum_from<2, I, G, PK>(g, vol_t, zyx_strides(g), r, count);
    return fp_ray_sum_from<0, I, G, PK>(g, vol, xyz_strides(g), r, count);
}

// Detector tile of a block of NW warps for the tunable projector variants:
// a warp covers WX x (32/WX) pixels (WX consecutive columns of 32/WX rows),
// the NW warps are stacked along the rows.  WX = 32, NW = 4 is tile_pixel.
template <int WX, int NW>
__device__ __forceinline__ bool tile_pixel_t(const GeomDev &g, int &i, int &j) {
    constexpr int WY = 32 / WX;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    i = blockIdx.x * WX + (lane % WX);
    j = (blockIdx.y * NW + w) * WY + lane / WX;
    return i < g.W && j < g.H;
}

// GenerateImage_MT (S/ImageFormationModel/TypicalRayProducer.core.h:168-224)
// for views [view0, view0 + gridDim.z).  T = float, or unsigned short for a
// BF16-stored volume (taps widened to FP32; the march and the sums are FP32).
// TX: the tile, samples in flight and corners of gather variant 10.
template <typename I, typename T, bool TX = false>
__global__ void __launch_bounds__(128) k_fp(const GeomDev g, const ViewRec *__restrict__ views,
                                            const T *__restrict__ vol, const T *__restrict__ vol_t,
                                            int view0, float *__restrict__ proj, float *__restrict__ raylen,
                                            float *__restrict__ weight, const FpTex tex) {
    int i, j;
    if (!tile_pixel_t<TX ? 8 : 32, 4>(g, i, j)) return;
    const int v = blockIdx.z;
    const ViewRec &vr = views[view0 + v];
    Ray r;
    make_ray(g, vr, i, j, r);
    int count = 0;
    const bool hit = r.tnear < r.tfar;
    float sum = 0.0f;
    if (hit) {
        if constexpr (TX)
            sum = fp_ray_sum_tex<8, true, T>(g, tex, r, &count);
        else
            sum = fp_ray_sum<I, sizeof(T) == 4 ? 2 : FP_GROUP>(g, vr, vol, vol_t, r, &count);  // (FP_DEFAULT_LOADS)
    }
    const size_t o = (size_t)v * g.W * g.H + i + (size_t)j * g.W;
    proj[o] = sum;
    if (raylen && hit) raylen[o] = r.tfar - r.tnear;
    if (weight) weight[o] = (float)count;
}

// Forward projection of one view with the SART correction as epilogue
// (ST_Tomography.cpp:667-676; Factor = 1 and pY == 0 in the reference, so
// c = (b - Ax) / (L + 1)).  L is the sticky ray length of the producer:
// updated where the ray hits, kept where it misses; with no state buffer
// (ray-based SART, whose producer is reset after every view) a miss gives L = 0.
// Tunable variants (fp_variant_name): the block's detector tile (WX, NW), the
// samples in flight per step (G) and whether pairs of samples share packed
// FP32x2 instructions (PK) change only which thread projects which ray, how
// far ahead its loads run and how many instructions carry the same roundings,
// never a ray's arithmetic.
// T, B: the storage of the volume and of the sinogram stack (float, or BF16
// bits widened exactly to FP32).
// TX: the corners come from the texture of `tex` (volumes below 2^31 voxels),
// not from vol and vol_t.
template <typename I, int WX = 32, int NW = 4, int G = FP_GROUP, bool PK = false, typename T = float,
          typename B = float, bool TX = false>
__global__ void __launch_bounds__(32 * NW) k_fp_corr(const GeomDev g, const ViewRec *__restrict__ views,
                                                     const T *__restrict__ vol, const T *__restrict__ vol_t,
                                                     const ViewSel sel, const B *__restrict__ b_stack,
                                                     float *__restrict__ raylen_state,
                                                     float *__restrict__ corr,
                                                     int skip_staged, const FpTex tex) {
    int i, j;
    if (!tile_pixel_t<WX, NW>(g, i, j)) return;
    int local;
    const int view = sel_view(sel, local);
    const B *b = b_stack + (size_t)local * g.W * g.H;
    const ViewRec &vr = views[view];
    if (skip_staged && view_staged<T>(vr)) return;  // the slab-staged kernel projects this view
    Ray r;
    make_ray(g, vr, i, j, r);
    const size_t pix = i + (size_t)j * g.W;
    float L, sum = 0.0f;
    if (r.tnear < r.tfar) {
        if constexpr (TX)
            sum = fp_ray_sum_tex<G, PK, T>(g, tex, r, nullptr);
        else
            sum = fp_ray_sum<I, G, PK>(g, vr, vol, vol_t, r, nullptr);
        L = r.tfar - r.tnear;
        if (raylen_state) raylen_state[pix] = L;
    } else {
        L = raylen_state ? raylen_state[pix] : 0.0f;
    }
    cudaTriggerProgrammaticLaunchCompletion();
    corr[pix] = __fdiv_rn(__fsub_rn(ld_voxel(b + pix), sum), __fadd_rn(L, 1.0f));
}

// Stand-alone SART correction (ST_Tomography.cpp:667-676) for the unfused
// per-view form: the ray lengths are the sticky state k_fp updated on hits.
template <typename B>
__global__ void k_correction(long long n, const B *__restrict__ b, const float *__restrict__ ax,
                             const float *__restrict__ raylen, float *__restrict__ corr) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x)
        corr[k] = __fdiv_rn(__fsub_rn(ld_voxel(b + k), ax[k]), __fadd_rn(raylen ? raylen[k] : 0.0f, 1.0f));
}

// z-fastest copy of an x-fastest volume: out[z + y*nz + x*nz*ny] = in[x + y*nx + z*nx*ny].
// One 64x64 (x, z) tile of one y plane per block of 32x8 threads, through
// shared memory.  Interior tiles move two elements per access (8-byte float2
// or 4-byte ushort2 rows) when nx and nz are even and both arrays aligned to
// a pair; edge tiles move one.
template <typename T>
struct Pair2;
template <>
struct Pair2<float> {
    typedef float2 type;
};
template <>
struct Pair2<unsigned short> {
    typedef ushort2 type;
};

template <typename T>
__device__ __forceinline__ void transpose_tile(int nx, int ny, int nz, const T *__restrict__ in,
                                               T *__restrict__ out) {
    typedef typename Pair2<T>::type P;
    __shared__ T tile[64][65];  // tile[z - z0][x - x0]
    const int x0 = blockIdx.x * 64, z0 = blockIdx.y * 64, y = blockIdx.z;
    const size_t nxy = (size_t)nx * ny, nzy = (size_t)nz * ny;
    const T *src = in + (size_t)y * nx + x0 + (size_t)z0 * nxy;
    T *dst = out + (size_t)y * nz + z0 + (size_t)x0 * nzy;
    const int tx = threadIdx.x;
    const bool pairs = x0 + 64 <= nx && z0 + 64 <= nz && !(nx & 1) && !(nz & 1) &&
                       !(((uintptr_t)in | (uintptr_t)out) % sizeof(P));
    if (pairs) {
#pragma unroll
        for (int r = threadIdx.y; r < 64; r += 8) {
            const P v = reinterpret_cast<const P *>(src + r * nxy)[tx];
            tile[r][2 * tx] = v.x;
            tile[r][2 * tx + 1] = v.y;
        }
        __syncthreads();
#pragma unroll
        for (int r = threadIdx.y; r < 64; r += 8) {
            P v;
            v.x = tile[2 * tx][r];
            v.y = tile[2 * tx + 1][r];
            reinterpret_cast<P *>(dst + r * nzy)[tx] = v;
        }
    } else {
        for (int r = threadIdx.y; r < 64; r += 8)
            for (int c = tx; c < 64; c += 32)
                if (x0 + c < nx && z0 + r < nz) tile[r][c] = src[c + r * nxy];
        __syncthreads();
        for (int r = threadIdx.y; r < 64; r += 8)
            for (int c = tx; c < 64; c += 32)
                if (x0 + r < nx && z0 + c < nz) dst[c + r * nzy] = tile[c][r];
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_transpose_xz(int nx, int ny, int nz, const T *__restrict__ in,
                                                      T *__restrict__ out) {
    transpose_tile(nx, ny, nz, in, out);
}

// The transpose, only if the selected view gathers from the z-fastest copy
// (the choice is read on the device, so a captured graph can hold it).
template <typename T>
__global__ void __launch_bounds__(256) k_transpose_for_view(int nx, int ny, int nz,
                                                            const ViewRec *__restrict__ views, const ViewSel sel,
                                                            const T *__restrict__ in, T *__restrict__ out,
                                                            bool staged_only) {
    int local;
    const ViewRec &v = views[sel_view(sel, local)];
    if (v.layout != 1 || (staged_only && !view_staged<T>(v))) return;
    transpose_tile(nx, ny, nz, in, out);
}

// A volume's slices to their places in its mirror, four elements a thread.
template <typename T>
__global__ void __launch_bounds__(256) k_mirror(int slice, int pitch, const T *__restrict__ vol, T *__restrict__ mirror) {
    const T *in = vol + (size_t)blockIdx.y * slice;
    T *out = mirror + (size_t)blockIdx.y * pitch;
    const int k0 = blockIdx.x * 1024 + threadIdx.x;
    T v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (k0 + 256 * q < slice) v[q] = in[k0 + 256 * q];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (k0 + 256 * q < slice) out[k0 + 256 * q] = v[q];
}

__global__ void k_fill_zero(long long n, float *__restrict__ p) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x)
        p[k] = 0.0f;
}

// 32-bit gather offsets when every voxel index fits.
bool small_volume(const GeomDev &g) { return (long long)g.nx * g.ny * g.nz < (1LL << 31); }

dim3 ray_grid(const GeomDev &g, int nviews) {
    return dim3((g.W + 31) / 32, (g.H + 3) / 4, nviews);
}

dim3 transpose_grid(const GeomDev &g) { return dim3((g.nx + 63) / 64, (g.nz + 63) / 64, g.ny); }

// The gather ceiling of the forward projector: each ray of one view takes as
// many samples as its clip length holds, at the projector's step from its
// entry point, with the projector's cell, 8-corner gather and trilinear
// interpolation (G = 4 samples' loads in flight, packed pairs when PK; the
// corners as tld4 gathers of texture `tex` when TX), and none of its march
// control (no segment splits, no per-sample bound, a plain sum).  No
// counterpart in the reference: a measurement of the rate the gathers alone
// reach on a volume, the on-chip roofline of the projectors.
template <int FAST, bool PK, bool TX = false>
__global__ void __launch_bounds__(128) k_gather_ceiling(const GeomDev g, const ViewRec *__restrict__ views, int view,
                                                        const float *__restrict__ src, unsigned long long tex,
                                                        float *__restrict__ out, int *__restrict__ count) {
    int i, j;
    if (!tile_pixel(g, i, j)) return;
    Ray r;
    make_ray(g, views[view], i, j, r);
    const size_t pix = i + (size_t)j * g.W;
    float sum = 0.0f;
    int n = 0;
    if (r.tnear < r.tfar) {
        const Strides st = FAST ? zyx_strides(g) : xyz_strides(g);
        n = min((int)((r.tfar - r.tnear) / g.sd) + 1, 1 << 22);
        float p[3], step[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            p[k] = __fmaf_rn(r.vu[k], r.tnear, r.vz[k]);  // explicit roundings: every instantiation alike
            step[k] = __fmul_rn(r.vu[k], g.sd);
        }
        constexpr int G = 4;
        int k = 0;
        for (; k + G <= n; k += G) {
            float q[G][3];
            FpCell c[G];
            float v[G][8];
#pragma unroll
            for (int s = 0; s < G; ++s)
#pragma unroll
                for (int a = 0; a < 3; ++a) q[s][a] = __fmaf_rn((float)s, step[a], p[a]);
#pragma unroll
            for (int a = 0; a < 3; ++a) p[a] = __fmaf_rn((float)G, step[a], p[a]);
            if constexpr (PK) {
#pragma unroll
                for (int s = 0; s < G; s += 2) fp_cell2(g, q[s], q[s + 1], c[s], c[s + 1]);
            } else {
#pragma unroll
                for (int s = 0; s < G; ++s) fp_cell(g, q[s], c[s]);
            }
#pragma unroll
            for (int s = 0; s < G; ++s) {
                if constexpr (TX)
                    fp_corners_tex(tex, g.nx, c[s], v[s]);
                else
                    fp_corners<FAST, int>(src, st, c[s], v[s]);
            }
            if constexpr (PK) {
#pragma unroll
                for (int s = 0; s < G; s += 2) {
                    const float2 t = trilerp2(v[s], v[s + 1], c[s], c[s + 1]);
                    sum = __fadd_rn(sum, __fadd_rn(t.x, t.y));
                }
            } else {  // the same additions as the packed form
#pragma unroll
                for (int s = 0; s < G; s += 2)
                    sum = __fadd_rn(sum, __fadd_rn(trilerp(v[s], c[s]), trilerp(v[s + 1], c[s + 1])));
            }
        }
        for (; k < n; ++k) {
            FpCell c;
            fp_cell(g, p, c);
            float v[8];
            if constexpr (TX)
                fp_corners_tex(tex, g.nx, c, v);
            else
                fp_corners<FAST, int>(src, st, c, v);
            sum = __fadd_rn(sum, trilerp(v, c));
#pragma unroll
            for (int a = 0; a < 3; ++a) p[a] = __fadd_rn(p[a], step[a]);
        }
    }
    out[pix] = __fmul_rn(sum, g.sd);
    if (count) count[pix] = n;
}

}  // namespace

int sm_count() {
    // multiProcessorCount of each device, read once per device (148 on B200)
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return 148;
    }
    if (!cached[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = 148;
        }
        cached[dev] = n;
    }
    return cached[dev];
}

int grid_stride_blocks(long long n, int threads) {
    long long b = (n + threads - 1) / threads;
    // grid-stride loops: at most 8 resident 256-thread blocks per SM (2048 threads)
    const long long cap = (long long)sm_count() * (2048 / (threads > 0 ? threads : 256));
    return (int)(b < cap ? (b < 1 ? 1 : b) : cap);
}

FpFrom fp_from(long long voxels, float row_pitch, int esize, bool own, const FpCall &c) {
    int all = 0, in[2][10] = {};  // in[l][k]: layout l, in the first k classes
    for (int l = 0; l < 2; ++l)
        for (int b = 0; b < 9; ++b) in[l][b + 1] = in[l][b] + c.views[l][b], all += c.views[l][b];
    // a call along an axis: every view within 25 degrees of it, three in four in the first `classes`
    const auto close = [&](int l, int classes) { return in[l][5] == all && 4 * in[l][classes] >= 3 * all; };
    const bool few = c.rays <= FP_SPLIT_RAYS;  // the split form, if from a texture
    // (the copy's launch alone)
    const bool tiny = !own && voxels < (1LL << 19) && c.rays >= 20000 && c.rays < 100000 && close(0, 2);
    if (esize == 2) {
        const bool slow_copy = voxels > (1LL << 24) && close(0, 4) && c.rays * 150 < voxels && !few;
        const bool coarse = close(0, 2) && row_pitch > 2.0f && c.rays >= 80000 && c.rays < 200000;
        return !own && (slow_copy || coarse || tiny) ? FpFrom::OwnTexture : FpFrom::Texture;
    }
    const bool past_l2 = voxels * 4 > 96000000;
    // (loads of odd rows do better off the axis than those of rows a power of two apart)
    const int fine = voxels < (1LL << 19) ? 5 : 4;
    const int classes = own ? (voxels < (1LL << 22) ? 2 : 3) : (row_pitch < 0.9f || row_pitch > 2.5f ? fine : 3);
    const bool many = c.rays >= 80000 && (!own || (voxels >= (1LL << 17) && (all >= 6 || c.rays >= 500000)));
    if (many && close(0, classes) && (!past_l2 || row_pitch > 2.5f)) return FpFrom::Loads;
    if (past_l2) return close(0, 1) && row_pitch > 3.5f ? FpFrom::OwnTexture : FpFrom::Texture;
    // (along x loads make the z-fastest copy)
    if (voxels >= (1LL << 18) && c.rays >= 700000 && c.rays * 10 >= voxels && close(1, 3)) return FpFrom::Loads;
    if (own) return FpFrom::Texture;
    if (close(0, 3)) return few && voxels <= (1LL << 23) && !tiny ? FpFrom::Texture : FpFrom::OwnTexture;
    const bool slow_copy = voxels > (1LL << 23) && c.rays * 20 < voxels && !few;
    return slow_copy && close(0, row_pitch < 2.0f ? 5 : 4) ? FpFrom::OwnTexture : FpFrom::Texture;
}

namespace {
template <typename T>
cudaError_t fp_any(const GeomDev &g, const ViewRec *views, const T *vol, const T *vol_t, int view0, int nviews,
                   float *proj, float *raylen, float *weight, cudaStream_t s, const FpTex *tex) {
    if (tex && tex->ok && tex->esize == (int)sizeof(T) && small_volume(g)) {
        if ((long long)g.W * g.H * nviews <= FP_SPLIT_RAYS)
            return launch_fp_split(g, views, view0, nviews, proj, raylen, weight, s, *tex);
        k_fp<int, T, true><<<dim3((g.W + 7) / 8, (g.H + 15) / 16, nviews), 128, 0, s>>>(g, views, vol, vol_t, view0, proj,
                                                                                      raylen, weight, *tex);
    } else if (small_volume(g)) {
        k_fp<int, T><<<ray_grid(g, nviews), 128, 0, s>>>(g, views, vol, vol_t, view0, proj, raylen, weight, FpTex{});
    } else {
        k_fp<long long, T><<<ray_grid(g, nviews), 128, 0, s>>>(g, views, vol, vol_t, view0, proj, raylen, weight,
                                                                FpTex{});
    }
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_fp(const GeomDev &g, const ViewRec *views, const float *vol, const float *vol_t, int view0,
                      int nviews, float *proj, float *raylen, float *weight, cudaStream_t s, const FpTex *tex) {
    return fp_any(g, views, vol, vol_t, view0, nviews, proj, raylen, weight, s, tex);
}

cudaError_t launch_fp(const GeomDev &g, const ViewRec *views, const unsigned short *vol, const unsigned short *vol_t,
                      int view0, int nviews, float *proj, float *raylen, float *weight, cudaStream_t s,
                      const FpTex *tex) {
    return fp_any(g, views, vol, vol_t, view0, nviews, proj, raylen, weight, s, tex);
}

namespace {

// One launch of gather variant <WX, NW, G, PK, TX>: a block is NW warps of WX x (32/WX) pixels.
template <int WX, int NW, int G, bool PK = false, bool TX = false>
void fp_corr_variant(const GeomDev &g, const ViewRec *views, const float *vol, const float *vol_t, const ViewSel &sel,
                     const float *b_stack, float *raylen_state, float *corr, cudaStream_t s,
                     int skip, const FpTex &tex = FpTex{}) {
    constexpr int TH = (32 / WX) * NW;  // detector rows per block
    k_fp_corr<int, WX, NW, G, PK, float, float, TX>
        <<<dim3((g.W + WX - 1) / WX, (g.H + TH - 1) / TH, 1), 32 * NW, 0, s>>>(
            g, views, vol, vol_t, sel, b_stack, raylen_state, corr, skip, tex);
}

// Device limits of pitch-linear 2D textures, read once per device.
struct TexLimits {
    int width = 0, height = 0, pitch = 0, pitch_align = 0, base_align = 0;
};

bool tex_limits(TexLimits &l) {
    static TexLimits cache[64];
    static bool have[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    if (!have[dev]) {
        TexLimits t;
        if (cudaDeviceGetAttribute(&t.width, cudaDevAttrMaxTexture2DLinearWidth, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&t.height, cudaDevAttrMaxTexture2DLinearHeight, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&t.pitch, cudaDevAttrMaxTexture2DLinearPitch, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&t.pitch_align, cudaDevAttrTexturePitchAlignment, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&t.base_align, cudaDevAttrTextureAlignment, dev) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        cache[dev] = t;
        have[dev] = true;
    }
    l = cache[dev];
    return true;
}

bool slices_fit(const TexLimits &l, const void *p, long long width, long long rows, long long pitch) {
    return p && width >= 2 && rows >= 2 && width <= l.width && rows <= l.height && pitch <= l.pitch &&
           !(l.pitch_align > 0 && pitch % l.pitch_align) && !(l.base_align > 0 && (uintptr_t)p % l.base_align);
}

// A point-sampled, clamped texture of `rows` rows of `width` texels over
// linear memory (FP32 texels, or 16-bit unsigned ones holding BF16 bits); 0
// where the limits do not admit it.
template <typename T>
unsigned long long slices_texture(const TexLimits &l, const T *p, long long width, long long rows, long long pitch) {
    if (!slices_fit(l, p, width, rows, pitch)) return 0;
    cudaResourceDesc rd{};
    rd.resType = cudaResourceTypePitch2D;
    rd.res.pitch2D.devPtr = const_cast<T *>(p);
    rd.res.pitch2D.desc = cudaCreateChannelDesc<T>();
    rd.res.pitch2D.width = (size_t)width;
    rd.res.pitch2D.height = (size_t)rows;
    rd.res.pitch2D.pitchInBytes = (size_t)pitch;
    cudaTextureDesc td{};
    td.addressMode[0] = td.addressMode[1] = cudaAddressModeClamp;
    td.filterMode = cudaFilterModePoint;
    td.readMode = cudaReadModeElementType;
    cudaTextureObject_t t = 0;
    if (cudaCreateTextureObject(&t, &rd, &td, nullptr) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (unsigned long long)t;
}

}  // namespace

const char *fp_variant_name(int v) {
    static const char *names[kFpVariants] = {"32x4 rays per block, 4 samples in flight",
                                             "32x2 rays per block, 4 in flight",
                                             "32x8 rays per block, 4 in flight",
                                             "warps of 16x2 rays, 16x8 per block, 4 in flight",
                                             "warps of 8x4 rays, 8x16 per block, 4 in flight",
                                             "32x4 rays per block, 2 in flight",
                                             "32x4 rays per block, 8 in flight",
                                             "32x4 rays per block, 4 in flight, packed pairs",
                                             "32x4 rays per block, 8 in flight, packed pairs",
                                             "32x8 rays per block, 4 in flight, packed pairs",
                                             "warps of 8x4 rays, 8x16 per block, 8 in flight, packed pairs, tld4 corners",
                                             "32x4 rays per block, 8 in flight, packed pairs, tld4 corners"};
    return v >= 0 && v < kFpVariants ? names[v] : "?";
}

bool is_tex_fp_variant(int fp_variant) { return fp_variant == 10 || fp_variant == 11; }

const char *fp16_variant_name(int v) {
    static const char *names[kFp16Variants] = {"32x4 rays per block, 4 samples in flight",
                                               "warps of 8x4 rays, 8 in flight, packed pairs, tld4 corners"};
    return v >= 0 && v < kFp16Variants ? names[v] : "?";
}

namespace {
template <typename T>
bool make_fp_tex_any(const GeomDev &g, const T *vol, FpTex &t, size_t pitch) {
    t = FpTex{};
    TexLimits l;
    if (!small_volume(g) || !tex_limits(l)) return false;
    const long long slice = (long long)g.nx * g.ny;
    t.x = slices_texture(l, vol, slice, g.nz, (pitch ? (long long)pitch : slice) * (long long)sizeof(T));
    t.ok = t.x != 0;
    t.esize = (int)sizeof(T);
    return t.ok != 0;
}
}  // namespace

bool make_fp_tex(const GeomDev &g, const float *vol, FpTex &t, size_t pitch) { return make_fp_tex_any(g, vol, t, pitch); }

bool make_fp_tex(const GeomDev &g, const unsigned short *vol, FpTex &t, size_t pitch) {
    return make_fp_tex_any(g, vol, t, pitch);
}

namespace {
template <typename T>
cudaError_t mirror_any(const GeomDev &g, const T *vol, T *mirror, cudaStream_t s) {
    const int slice = g.nx * g.ny;  // (a mirrored volume has fewer than 2^31 voxels)
    const int nb = (slice + 1023) / 1024;
    k_mirror<T><<<dim3(nb, g.nz), 256, 0, s>>>(slice, (int)fp_mirror_pitch(slice), vol, mirror);
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_mirror(const GeomDev &g, const float *vol, float *mirror, cudaStream_t s) {
    return mirror_any(g, vol, mirror, s);
}

cudaError_t launch_mirror(const GeomDev &g, const unsigned short *vol, unsigned short *mirror, cudaStream_t s) {
    return mirror_any(g, vol, mirror, s);
}

bool fp_tex_fits(const GeomDev &g, const void *vol, int esize, size_t pitch) {
    TexLimits l;
    const long long slice = (long long)g.nx * g.ny;
    return small_volume(g) && tex_limits(l) && slices_fit(l, vol, slice, g.nz, (pitch ? (long long)pitch : slice) * esize);
}

bool fp_tex_admits(const GeomDev &g, int esize) {
    const void *aligned = reinterpret_cast<const void *>((uintptr_t)4096);  // (as cudaMalloc's)
    return fp_tex_fits(g, aligned, esize) || fp_tex_fits(g, aligned, esize, fp_mirror_pitch((size_t)g.nx * g.ny));
}

void destroy_fp_tex(FpTex &t) {
    if (t.x) cudaDestroyTextureObject((cudaTextureObject_t)t.x);
    t = FpTex{};
}

cudaError_t launch_fp_corr(const GeomDev &g, const ViewRec *views, const float *vol, const float *vol_t,
                           const ViewSel &sel, const float *b_stack, float *raylen_state, float *corr,
                           cudaStream_t s, const FpSlabMaps *maps, int *status,
                           int fp_variant, const FpTex *tex, int chains) {
    const int skip = maps && maps->ok && maps->esize == 4 && (!vol_t || maps->has_z);
    // a texture variant without a usable texture runs the load-based variant of the same shape
    if (is_tex_fp_variant(fp_variant) && !(tex && tex->ok && tex->esize == 4)) fp_variant = fp_variant == 10 ? 4 : 8;
    const FpTex tx = tex ? *tex : FpTex{};
    if (skip) {
        cudaError_t e = launch_fp_corr_slab(g, views, *maps, vol, vol_t, sel, b_stack, raylen_state, corr, s,
                                            status);
        if (e != cudaSuccess) return e;
    }
    if (!small_volume(g)) {
        k_fp_corr<long long><<<ray_grid(g, 1), 128, 0, s>>>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr,
                                                            skip, FpTex{});
        return cudaGetLastError();
    }
    if (is_tex_fp_variant(fp_variant) && (long long)g.W * g.H <= fp_split_rays(chains))
        return launch_fp_corr_split(g, views, sel, b_stack, raylen_state, corr, s, tx, skip);
    switch (fp_variant) {
    case 1: fp_corr_variant<32, 2, 4>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s, skip); break;
    case 2: fp_corr_variant<32, 8, 4>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s, skip); break;
    case 3: fp_corr_variant<16, 4, 4>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s, skip); break;
    case 4: fp_corr_variant<8, 4, 4>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s, skip); break;
    case 5: fp_corr_variant<32, 4, 2>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s, skip); break;
    case 6: fp_corr_variant<32, 4, 8>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s, skip); break;
    case 7: fp_corr_variant<32, 4, 4, true>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s, skip); break;
    case 8: fp_corr_variant<32, 4, 8, true>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s, skip); break;
    case 9: fp_corr_variant<32, 8, 4, true>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s, skip); break;
    case 10:
        fp_corr_variant<8, 4, 8, true, true>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s,
                                             skip, tx);
        break;
    case 11:
        fp_corr_variant<32, 4, 8, true, true>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s,
                                              skip, tx);
        break;
    default: fp_corr_variant<32, 4, 4>(g, views, vol, vol_t, sel, b_stack, raylen_state, corr, s, skip); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_transpose(const GeomDev &g, const float *in, float *out, cudaStream_t s) {
    k_transpose_xz<float><<<transpose_grid(g), dim3(32, 8), 0, s>>>(g.nx, g.ny, g.nz, in, out);
    return cudaGetLastError();
}

cudaError_t launch_transpose_bf16(const GeomDev &g, const unsigned short *in, unsigned short *out, cudaStream_t s) {
    k_transpose_xz<unsigned short><<<transpose_grid(g), dim3(32, 8), 0, s>>>(g.nx, g.ny, g.nz, in, out);
    return cudaGetLastError();
}

cudaError_t launch_transpose_for_view(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *in,
                                      float *out, cudaStream_t s, bool staged_only) {
    k_transpose_for_view<float><<<transpose_grid(g), dim3(32, 8), 0, s>>>(g.nx, g.ny, g.nz, views, sel, in, out,
                                                                         staged_only);
    return cudaGetLastError();
}

cudaError_t launch_transpose_for_view(const GeomDev &g, const ViewRec *views, const ViewSel &sel,
                                      const unsigned short *in, unsigned short *out, cudaStream_t s,
                                      bool staged_only) {
    k_transpose_for_view<unsigned short><<<transpose_grid(g), dim3(32, 8), 0, s>>>(g.nx, g.ny, g.nz, views, sel, in,
                                                                                  out, staged_only);
    return cudaGetLastError();
}

cudaError_t launch_correction(long long n, const float *b, const float *ax, const float *raylen,
                              float *corr, cudaStream_t s) {
    k_correction<float><<<grid_stride_blocks(n, 256), 256, 0, s>>>(n, b, ax, raylen, corr);
    return cudaGetLastError();
}

cudaError_t launch_correction(long long n, const unsigned short *b, const float *ax, const float *raylen,
                              float *corr, cudaStream_t s) {
    k_correction<unsigned short><<<grid_stride_blocks(n, 256), 256, 0, s>>>(n, b, ax, raylen, corr);
    return cudaGetLastError();
}

cudaError_t launch_fp_corr(const GeomDev &g, const ViewRec *views, const unsigned short *vol,
                           const unsigned short *vol_t, const ViewSel &sel, const unsigned short *b_stack,
                           float *raylen_state, float *corr, cudaStream_t s,
                           const FpSlabMaps *maps, int *status, int fp_variant16, const FpTex *tex, int chains) {
    typedef unsigned short U;
    const int skip = maps && maps->ok && maps->esize == 2 && (!vol_t || maps->has_z);
    if (skip) {
        cudaError_t e = launch_fp_corr_slab(g, views, *maps, vol, vol_t, sel, b_stack, raylen_state, corr, s,
                                            status);
        if (e != cudaSuccess) return e;
    }
    if (fp_variant16 == 1 && tex && tex->ok && tex->esize == 2 && small_volume(g)) {
        const FpTex tx = *tex;
        if ((long long)g.W * g.H <= fp_split_rays(chains))
            return launch_fp_corr_split(g, views, sel, b_stack, raylen_state, corr, s, tx, skip);
        constexpr int WX = 8, NW = 4, TH = (32 / WX) * NW;
        k_fp_corr<int, WX, NW, 8, true, U, U, true><<<dim3((g.W + WX - 1) / WX, (g.H + TH - 1) / TH, 1), 32 * NW, 0, s>>>(
            g, views, vol, vol_t, sel, b_stack, raylen_state, corr, skip, tx);
        return cudaGetLastError();
    }
    if (small_volume(g))
        k_fp_corr<int, 32, 4, FP_GROUP, false, U, U><<<ray_grid(g, 1), 128, 0, s>>>(
            g, views, vol, vol_t, sel, b_stack, raylen_state, corr, skip, FpTex{});
    else
        k_fp_corr<long long, 32, 4, FP_GROUP, false, U, U><<<ray_grid(g, 1), 128, 0, s>>>(
            g, views, vol, vol_t, sel, b_stack, raylen_state, corr, skip, FpTex{});
    return cudaGetLastError();
}

cudaError_t launch_gather_ceiling(const GeomDev &g, const ViewRec *views, const ViewRec &host_view, int view,
                                  const float *vol, const float *vol_t, int packed, float *out, int *count,
                                  cudaStream_t s, const FpTex *tex) {
    if (!small_volume(g)) return cudaErrorInvalidValue;
    if (tex) {  // packed pairs, tld4 corners
        if (!tex->ok) return cudaErrorInvalidValue;
        k_gather_ceiling<0, true, true><<<ray_grid(g, 1), 128, 0, s>>>(g, views, view, vol, tex->x, out, count);
        return cudaGetLastError();
    }
    const bool zf = vol_t && host_view.layout == 1;
    const float *src = zf ? vol_t : vol;
    if (zf && packed) k_gather_ceiling<2, true><<<ray_grid(g, 1), 128, 0, s>>>(g, views, view, src, 0, out, count);
    else if (zf) k_gather_ceiling<2, false><<<ray_grid(g, 1), 128, 0, s>>>(g, views, view, src, 0, out, count);
    else if (packed) k_gather_ceiling<0, true><<<ray_grid(g, 1), 128, 0, s>>>(g, views, view, src, 0, out, count);
    else k_gather_ceiling<0, false><<<ray_grid(g, 1), 128, 0, s>>>(g, views, view, src, 0, out, count);
    return cudaGetLastError();
}

cudaError_t launch_fill_zero(float *p, long long n, cudaStream_t s) {
    k_fill_zero<<<grid_stride_blocks(n, 256), 256, 0, s>>>(n, p);
    return cudaGetLastError();
}

}  // namespace stt
