// k_scatter.cu -- the scatters: the ray-driven backprojection
// (S/ST_Tomo/ST_Tomography.cpp:733-764, S/ImageFormationModel/
// SingleScalarVolume.core.h:73-84, 128-143) and the exact adjoint A^T of the
// forward projector.
//
// Both march every ray as the projector does and add to the 8 corners of every
// sample with float atomics, whose rate at L2 bounds them: it counts the sectors a
// warp's atomics touch.  Neighbouring detector rows' rays lie a fraction of a voxel
// apart, so a thread marches R of them in step and adds those that share a cell
// column in registers before they go to memory (scatter_column).  The lanes stay
// in step too: one that ran ahead would split the warp's atomics.
// Per view with the update, us, views at 0 / 45 / 90 degrees, a ray a thread -> R:
// 256^3 / 512^2 609/902/974 -> 437/597/643 (R = 4; 455/662/750 with 2, 502/694/590
// with 6), 192^3 / 256^2 145/220/224 -> 150/233/193 (R = 2); the adjoint of those
// and a fourth view 2382 -> 1309, 504 -> 425.  Measured and not kept: lanes 2, 4 or 8
// columns apart, whose atomics never meet (426/688/655 to 562/699/610 with R = 4:
// meeting costs less than the sectors); z-fastest accumulators for the views along
// x (the scatter 576 -> 370 us at 90 degrees, but emptying 200 MB of them across the
// volume's order takes 820 us, in order 70).
#include <algorithm>

#include "stt_internal.cuh"
#include "stt_kernels.h"

namespace stt {

namespace {

constexpr int THREADS = 128;
constexpr float CLOSE_ROWS = 0.75f;  // voxels between rows that four rays a thread pay for

// What a march adds to a voxel: (c w, w) to the interleaved accumulators of the
// ray-driven backprojection, or c w to the adjoint's volume.  A Row holds the
// sums of the four corners of one y: (x, z), (x+1, z), (x, z+1), (x+1, z+1).
struct PairSink {
    static constexpr bool SKIP_ZERO = false;  // (a ray of zero correction still adds its weights)
    float2 *acc;
    struct Row {
        float c[4], w[4];
    };
    static __device__ __forceinline__ void clear(Row &r) {
#pragma unroll
        for (int m = 0; m < 4; ++m) r.c[m] = r.w[m] = 0.0f;
    }
    static __device__ __forceinline__ void add(Row &r, const float w[4], float f, float c) {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const float q = w[m] * f;
            r.w[m] += q;
            r.c[m] = fmaf(c, q, r.c[m]);
        }
    }
    // x-neighbours are adjacent; where the first is 16-byte aligned they go as one
    // vector atomic
    __device__ __forceinline__ void flush(const Row &r, size_t o, size_t slice) const {
#pragma unroll
        for (int m = 0; m < 4; m += 2) {
            float2 *p = acc + o + (m ? slice : 0);
            if (!(reinterpret_cast<uintptr_t>(p) & 15)) {
                atomicAdd(reinterpret_cast<float4 *>(p), make_float4(r.c[m], r.w[m], r.c[m + 1], r.w[m + 1]));
            } else {
                atomicAdd(p, make_float2(r.c[m], r.w[m]));
                atomicAdd(p + 1, make_float2(r.c[m + 1], r.w[m + 1]));
            }
        }
    }
};

struct ValueSink {
    static constexpr bool SKIP_ZERO = true;
    float *vol;
    struct Row {
        float c[4];
    };
    static __device__ __forceinline__ void clear(Row &r) {
#pragma unroll
        for (int m = 0; m < 4; ++m) r.c[m] = 0.0f;
    }
    static __device__ __forceinline__ void add(Row &r, const float w[4], float f, float c) {
#pragma unroll
        for (int m = 0; m < 4; ++m) r.c[m] = fmaf(c, w[m] * f, r.c[m]);
    }
    __device__ __forceinline__ void flush(const Row &r, size_t o, size_t slice) const {
#pragma unroll
        for (int m = 0; m < 4; m += 2) {
            float *p = vol + o + (m ? slice : 0);
            if (!(reinterpret_cast<uintptr_t>(p) & 7)) {  // (the caller's array may start anywhere on 4 bytes)
                atomicAdd(reinterpret_cast<float2 *>(p), make_float2(r.c[m], r.c[m + 1]));
            } else {
                atomicAdd(p, r.c[m]);
                atomicAdd(p + 1, r.c[m + 1]);
            }
        }
    }
};

// A ray's march state between its segments (shared memory, a column per thread).
enum { VZ = 0, VU = 3, TNEAR = 6, TFAR, TMAX, T1 = TMAX + 3, BUDGET, COLD };

// R rays of one detector column, rows j0 .. j0+R-1, marched in step: the
// samples of march() in stt_internal.cuh.  Every lane of the warp calls this.
template <int R, typename Sink>
__device__ __forceinline__ void scatter_column(const GeomDev &g, const ViewRec &vr, int i, int j0,
                                               const float (&value)[R], const Sink &sink,
                                               float (*cold)[COLD][THREADS]) {
    const int tid = threadIdx.x;
    const float hx = (float)(g.nx - 1), hy = (float)(g.ny - 1), hz = (float)(g.nz - 1), sd = g.sd;
    const size_t slice = (size_t)g.nx * g.ny;
    float t[R], px[R], py[R], pz[R], tb[R], sx[R], sy[R], sz[R], c[R];
    int left[R];  // samples the segment may still hold; 0: at its end; -1: the ray is done
#pragma unroll
    for (int r = 0; r < R; ++r) {
        c[r] = value[r];
        left[r] = -1;
        t[r] = tb[r] = px[r] = py[r] = pz[r] = sx[r] = sy[r] = sz[r] = 0.0f;
        if (i < g.W && j0 + r < g.H) {
            Ray ray;
            make_ray(g, vr, i, j0 + r, ray);
            if (ray.tnear < ray.tfar && !(Sink::SKIP_ZERO && c[r] == 0.0f)) {
                MarchDda d;
                float p[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) p[k] = __fadd_rn(ray.vz[k], __fmul_rn(ray.vu[k], ray.tnear));
                march_dda(g, ray, p, d);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    cold[r][VZ + k][tid] = ray.vz[k];
                    cold[r][VU + k][tid] = ray.vu[k];
                    cold[r][TMAX + k][tid] = d.tmax[k];
                }
                cold[r][TNEAR][tid] = cold[r][T1][tid] = ray.tnear;
                cold[r][TFAR][tid] = ray.tfar;
                cold[r][BUDGET][tid] = __int_as_float(1 << 22);
                sx[r] = d.step[0], sy[r] = d.step[1], sz[r] = d.step[2];
                // the entry sample: a segment of one before the march's
                px[r] = p[0], py[r] = p[1], pz[r] = p[2];
                left[r] = 1;
                tb[r] = 1.0f;
            }
        }
    }
    float dt = 1.0f;  // (past the entry sample's segment; then the sample distance)
    while (true) {
        bool any = false;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            // the next segment that holds a sample
            while (left[r] >= 0 && !(left[r] > 0 && t[r] < tb[r])) {
                const float t1 = cold[r][T1][tid], tfar = cold[r][TFAR][tid], tnear = cold[r][TNEAR][tid];
                const int budget = __float_as_int(cold[r][BUDGET][tid]);
                float m0 = cold[r][TMAX][tid], m1 = cold[r][TMAX + 1][tid], m2 = cold[r][TMAX + 2][tid];
                if (!(t1 < tfar) || budget <= 0) {
                    left[r] = -1;
                    break;
                }
                float b = rmin(rmin(m0, m1), m2);
                if (b > tfar) b = tfar;
                const float s = __fadd_rn(__fmul_rn(ceilf(__fdiv_rn(__fsub_rn(t1, tnear), sd)), sd), tnear);
                const int cap = (int)fminf(ceilf(__fdiv_rn(b - s, sd)) + 2.0f, (float)budget);
                cold[r][BUDGET][tid] = __int_as_float(budget - (cap > 0 ? cap : 0));
                t[r] = s;
                tb[r] = b;
                px[r] = __fadd_rn(cold[r][VZ][tid], __fmul_rn(cold[r][VU][tid], s));
                py[r] = __fadd_rn(cold[r][VZ + 1][tid], __fmul_rn(cold[r][VU + 1][tid], s));
                pz[r] = __fadd_rn(cold[r][VZ + 2][tid], __fmul_rn(cold[r][VU + 2][tid], s));
                left[r] = cap > 0 ? cap : 0;
                // the axis just split does not split again: its next split lies a
                // whole volume on, past the ray's end
                if (m0 < m1) {
                    if (m0 < m2) m0 = INFINITY;
                    else m2 = INFINITY;
                } else {
                    if (m1 < m2) m1 = INFINITY;
                    else m2 = INFINITY;
                }
                cold[r][TMAX][tid] = m0, cold[r][TMAX + 1][tid] = m1, cold[r][TMAX + 2][tid] = m2;
                cold[r][T1][tid] = b;
            }
            any |= left[r] > 0;
        }
        if (!__any_sync(0xffffffffu, any)) break;
        // One sample of every ray, from the lowest row up.  Rays whose samples
        // share the (x, z) cell add into the same two rows of sums; a row goes to
        // memory when the next ray's cell has left it.
        typename Sink::Row lo, hi;
        Sink::clear(lo);
        Sink::clear(hi);
        size_t at = 0;  // the lower row's first corner
        int cy = -1, cxz = -1;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (left[r] > 0) {
                const float qx = fmaxf(fminf(px[r], hx), 0.0f), qy = fmaxf(fminf(py[r], hy), 0.0f),
                            qz = fmaxf(fminf(pz[r], hz), 0.0f);
                const int ix = min((int)qx, g.nx - 2), iy = min((int)qy, g.ny - 2), iz = min((int)qz, g.nz - 2);
                const float fx = qx - (float)ix, fy = qy - (float)iy, fz = qz - (float)iz;
                const int xz = ix + g.nx * iz;
                const bool same = xz == cxz;
                if (cy >= 0 && !(same && iy == cy)) {
                    sink.flush(lo, at, slice);
                    if (same && iy == cy + 1) {
                        lo = hi;
                    } else {
                        sink.flush(hi, at + g.nx, slice);
                        Sink::clear(lo);
                    }
                    Sink::clear(hi);
                }
                cy = iy, cxz = xz;
                at = ix + (size_t)iy * g.nx + (size_t)iz * slice;
                const float gx = 1.0f - fx, gz = 1.0f - fz;
                const float w[4] = {gx * gz, fx * gz, gx * fz, fx * fz};
                Sink::add(lo, w, 1.0f - fy, c[r]);
                Sink::add(hi, w, fy, c[r]);
                --left[r];
                t[r] = __fadd_rn(t[r], dt);
                px[r] = __fadd_rn(px[r], sx[r]);
                py[r] = __fadd_rn(py[r], sy[r]);
                pz[r] = __fadd_rn(pz[r], sz[r]);
            }
        }
        if (cy >= 0) {
            sink.flush(lo, at, slice);
            sink.flush(hi, at + g.nx, slice);
        }
        dt = sd;
    }
}

// The most rays a thread that the distance of the rows pays for.
int most_rays(const GeomDev &g) {
    if (!((long long)g.nx * g.nz < (1LL << 31))) return 1;  // (32-bit cell keys)
    return g.row_pitch < CLOSE_ROWS ? 4 : g.row_pitch < 1.05f ? 2 : 1;
}

// Rays a thread: enough to merge where rows lie close, as long as the launch
// still fills the GPU.  Backprojection of one view with 1 / 2 / 4, us, mean of six
// views: rows 0.6 voxels apart 65,536 rays 130/129/193, 102,400 226/208/256,
// 147,456 363/289/308, 200,704 575/439/417; 0.9 apart 65,536 205/203/287, 90,000
// 319/304/381; 1.2 apart (128^2 at 128^3) 52/99.
int merged_rays(const GeomDev &g, int nviews) {
    const long long rays = (long long)g.W * g.H * nviews;
    const int most = most_rays(g);
    if (most == 4 && rays >= 180000) return 4;
    return most > 1 && rays >= 90000 ? 2 : 1;
}

// The adjoint of a residual that is nowhere zero the same, for all views of the launch.
// But its rays of zero residual are skipped, and what fills the GPU is the
// others: some 20 % where an object's shadow is surrounded by nothing.  So a launch
// needs several times as many.  Its time with 1 / 2 / 4, us, residuals dense / live in
// one ellipse of 20 % / in spots of 9 x 9 on 16 %, volume cold in the L2 (hot the same
// within 5 %):
//   rows 0.6 apart  128^3 4 x 256^2   342/254/244  188/135/186   96/106/160
//                   256^3 1 x 512^2   453/356/338  211/168/283  161/197/287
//                         2 x 512^2   922/680/557  338/281/344  254/283/363
//                         4 x 512^2  2446/1624/1350  782/639/610  465/432/557
//                        12 x 512^2  6822/4498/3397 2082/1491/1298 1223/1071/1302
//   rows 0.9 apart  192x176x160 2 x 256x240  174/139/190   63/109/180   74/107/174
//                   4              408/350/389  234/190/207  115/141/203
//                  12            1006/801/797   444/424/449  217/256/338
//                  24           1864/1416/1234  732/619/696  377/410/508
//                   256^3 1 x 341^2   229/195/293   92/154/272  106/174/274
//                        12 x 341^2  3092/2315/1987 1026/905/909 580/588/771
// and of objects' shadows (16 to 20 % live): 80^3 11 x 132x106 101/95, 100^3 1 x 121x153
// 47/77, 160^3 2 x 256^2 64/105, 4 x 256^2 187/163, 176^3 6 x 184x187 136/185,
// 192x176x160 12 x 256x240 407/399.  A longer ray takes more other rays to hide, so two
// rays a thread take 1500 of them per voxel of the largest extent and 150,000 at least;
// past that line the spots, which no scan leaves, lose 18 % at most, the others gain.
int merged_rays_adjoint(const GeomDev &g, int nviews) {
    const long long rays = (long long)g.W * g.H * nviews;
    const int most = most_rays(g), extent = std::max(g.nx, std::max(g.ny, g.nz));
    if (most == 1 || rays < std::max(150000LL, 1500LL * extent)) return 1;
    return most == 4 && rays >= 3000000 ? 4 : 2;
}

// BP-mode march (SingleScalarVolume.core.h:128-143, UpdateContributionSum
// :73-84): every sample adds (c*w_k, w_k) to its 8 clamped corners.
template <int R>
__global__ void __launch_bounds__(THREADS) k_bp_ray_scatter(const GeomDev g, const ViewRec *__restrict__ views,
                                                           const ViewSel sel, const float *__restrict__ corr,
                                                           float2 *__restrict__ acc) {
    __shared__ float cold[R][COLD][THREADS];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j0 = (blockIdx.y * (THREADS / 32) + (threadIdx.x >> 5)) * R;
    int local;
    const ViewRec &vr = views[sel_view(sel, local)];
    float c[R];
#pragma unroll
    for (int r = 0; r < R; ++r) c[r] = i < g.W && j0 + r < g.H ? __ldg(corr + i + (size_t)(j0 + r) * g.W) : 0.0f;
    scatter_column<R>(g, vr, i, j0, c, PairSink{acc}, cold);
}

// The same with a ray a thread: views of few rays, or rows a voxel apart.
__global__ void __launch_bounds__(THREADS) k_bp_ray_scatter_1(const GeomDev g, const ViewRec *__restrict__ views,
                                                             const ViewSel sel, const float *__restrict__ corr,
                                                             float2 *__restrict__ acc) {
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = blockIdx.y * (THREADS / 32) + (threadIdx.x >> 5);
    if (i >= g.W || j >= g.H) return;
    int local;
    const ViewRec &vr = views[sel_view(sel, local)];
    Ray r;
    make_ray(g, vr, i, j, r);
    if (!(r.tnear < r.tfar)) return;
    const float c = __ldg(corr + i + (size_t)j * g.W);
    march(g, r, [&](const float p[3]) {
        Taps t;
        make_taps(g, p, t);
        float w[8];
        tri_weights(t, w);
        scatter_corners(acc, t, c, w);
    });
}

// Exact adjoint of k_fp: vol_bar[corner] += sd * w_k * y for every sample,
// the entry sample twice, clamped corners collapsing as in the forward pass.
template <int R>
__global__ void __launch_bounds__(THREADS) k_fp_adjoint(const GeomDev g, const ViewRec *__restrict__ views, int view0,
                                                       const float *__restrict__ proj_bar, float *__restrict__ vol_bar) {
    __shared__ float cold[R][COLD][THREADS];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j0 = (blockIdx.y * (THREADS / 32) + (threadIdx.x >> 5)) * R;
    const float *y = proj_bar + (size_t)blockIdx.z * g.W * g.H + i;
    float c[R];
#pragma unroll
    for (int r = 0; r < R; ++r) c[r] = i < g.W && j0 + r < g.H ? __ldg(y + (size_t)(j0 + r) * g.W) * g.sd : 0.0f;
    scatter_column<R>(g, views[view0 + blockIdx.z], i, j0, c, ValueSink{vol_bar}, cold);
}

__global__ void __launch_bounds__(THREADS) k_fp_adjoint_1(const GeomDev g, const ViewRec *__restrict__ views, int view0,
                                                         const float *__restrict__ proj_bar,
                                                         float *__restrict__ vol_bar) {
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = blockIdx.y * (THREADS / 32) + (threadIdx.x >> 5);
    if (i >= g.W || j >= g.H) return;
    const int v = blockIdx.z;
    const float y = __ldg(proj_bar + (size_t)v * g.W * g.H + i + (size_t)j * g.W);
    if (y == 0.0f) return;
    Ray r;
    make_ray(g, views[view0 + v], i, j, r);
    if (!(r.tnear < r.tfar)) return;
    const float ys = y * g.sd;
    march(g, r, [&](const float p[3]) {
        Taps t;
        make_taps(g, p, t);
        float w[8];
        tri_weights(t, w);
        // x-neighbour corners inside the volume whose first address is 8-byte
        // aligned (the caller's vol_bar may start anywhere on 4 bytes): one
        // vector atomic (the same terms)
#pragma unroll
        for (int m = 0; m < 8; m += 2) {
            const long long idx = tap_index(t, m);
            if (t.dx == 1 && !(reinterpret_cast<uintptr_t>(vol_bar + idx) & 7)) {
                atomicAdd(reinterpret_cast<float2 *>(vol_bar + idx), make_float2(ys * w[m], ys * w[m + 1]));
            } else {
                atomicAdd(vol_bar + idx, ys * w[m]);
                atomicAdd(vol_bar + idx + t.dx, ys * w[m + 1]);
            }
        }
    });
}

// Ray-BP normalisation (ST_Tomography.cpp:746-762): vol += contrib/weight,
// clamped with the reference macros so 0/0 = NaN becomes 0; the accumulator
// is reset for the next view (TypicalRayProducer::Initial, TypicalRayProducer.cpp:91-95).
template <typename T>
__global__ void k_bp_ray_update(long long n, float2 *__restrict__ acc, T *__restrict__ vol, float gmax) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        float2 a = acc[k];
        float v = ld_stored(vol + k) + __fdiv_rn(a.x, a.y);
        st_stored(vol + k, rmax(rmin(gmax, v), 0.0f));
        acc[k] = make_float2(0.0f, 0.0f);
    }
}

// Adds the scatter accumulators to caller arrays and clears them: the raw
// contributions and weights of the reference's backprojection mode
// (SingleScalarVolume.core.h:128-143, read back through
// TypicalRayProducer::GetContributions / GetTotalWeight).
__global__ void k_acc_split(long long n, float2 *__restrict__ acc, float *__restrict__ contrib,
                            float *__restrict__ wsum) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        const float2 a = acc[k];
        contrib[k] += a.x;
        wsum[k] += a.y;
        acc[k] = make_float2(0.0f, 0.0f);
    }
}

bool small_volume(const GeomDev &g) { return (long long)g.nx * g.ny * g.nz < (1LL << 31); }

dim3 column_grid(const GeomDev &g, int rays, int nviews) {
    const int rows = THREADS / 32 * rays;
    return dim3((g.W + 31) / 32, (g.H + rows - 1) / rows, nviews);
}

// The scatter of the ray-driven backprojection: ray variant 1 (the slab box,
// below 2^31 voxels) or 0 (atomics to memory, rows merged).
cudaError_t scatter(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr, float2 *acc,
                    cudaStream_t s, int ray_variant) {
    if (ray_variant < 0) ray_variant = default_ray_variant(g);
    if (ray_variant == 1 && small_volume(g)) return launch_bp_ray_scatter_slab(g, views, sel, corr, acc, s);
    const int rays = merged_rays(g, 1);
    const dim3 grid = column_grid(g, rays, 1);
    if (rays == 4) k_bp_ray_scatter<4><<<grid, THREADS, 0, s>>>(g, views, sel, corr, acc);
    else if (rays == 2) k_bp_ray_scatter<2><<<grid, THREADS, 0, s>>>(g, views, sel, corr, acc);
    else k_bp_ray_scatter_1<<<grid, THREADS, 0, s>>>(g, views, sel, corr, acc);
    return cudaGetLastError();
}

template <typename T>
cudaError_t bp_ray_any(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr, float2 *acc,
                       T *vol, float gmax, cudaStream_t s, int ray_variant) {
    const cudaError_t e = scatter(g, views, sel, corr, acc, s, ray_variant);
    if (e != cudaSuccess) return e;
    const long long n = (long long)g.nx * g.ny * g.nz;
    k_bp_ray_update<T><<<grid_stride_blocks(n, 256), 256, 0, s>>>(n, acc, vol, gmax);
    return cudaGetLastError();
}

}  // namespace

int adjoint_rays(const GeomDev &g, int nviews, bool dense) {
    return dense ? merged_rays(g, nviews) : merged_rays_adjoint(g, nviews);
}

const char *ray_variant_name(int v) {
    static const char *names[kRayVariants] = {"global vector atomics, neighbouring rows merged",
                                              "shared-memory box per slab"};
    return v >= 0 && v < kRayVariants ? names[v] : "?";
}

// Atomics to memory, but for large volumes whose detector rows lie too far apart
// to merge.  Per view with the update, us, 0 / 45 / 90 degrees, atomics and box:
// 512^3 / 1024^2 2690/3681/4168 and 6428/7429/6659, 416^3 / 832^2 1581/2127/2283 and
// 3496/4171/3613, rows 1.2 voxels apart 512^3 / 512^2 1807/3762/5989 and
// 2092/3256/2752, 400^3 / 400^2 892/1269/2021 and 1109/1460/1223.
int default_ray_variant(const GeomDev &g) {
    return (long long)g.nx * g.ny * g.nz >= (1LL << 26) && g.row_pitch >= CLOSE_ROWS ? 1 : 0;
}

cudaError_t launch_bp_ray(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                          float2 *acc, float *vol, float gmax, cudaStream_t s, int ray_variant) {
    return bp_ray_any(g, views, sel, corr, acc, vol, gmax, s, ray_variant);
}

cudaError_t launch_bp_ray(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                          float2 *acc, unsigned short *vol, float gmax, cudaStream_t s, int ray_variant) {
    return bp_ray_any(g, views, sel, corr, acc, vol, gmax, s, ray_variant);
}

cudaError_t launch_bp_ray_scatter(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                                  float2 *acc, float *contrib, float *wsum, cudaStream_t s, int ray_variant) {
    const cudaError_t e = scatter(g, views, sel, corr, acc, s, ray_variant);
    if (e != cudaSuccess) return e;
    const long long n = (long long)g.nx * g.ny * g.nz;
    k_acc_split<<<grid_stride_blocks(n, 256), 256, 0, s>>>(n, acc, contrib, wsum);
    return cudaGetLastError();
}

cudaError_t launch_fp_adjoint(const GeomDev &g, const ViewRec *views, int view0, int nviews,
                              const float *proj_bar, float *vol_bar, cudaStream_t s, bool dense) {
    const int rays = adjoint_rays(g, nviews, dense);
    const dim3 grid = column_grid(g, rays, nviews);
    if (rays == 4) k_fp_adjoint<4><<<grid, THREADS, 0, s>>>(g, views, view0, proj_bar, vol_bar);
    else if (rays == 2) k_fp_adjoint<2><<<grid, THREADS, 0, s>>>(g, views, view0, proj_bar, vol_bar);
    else k_fp_adjoint_1<<<grid, THREADS, 0, s>>>(g, views, view0, proj_bar, vol_bar);
    return cudaGetLastError();
}

}  // namespace stt
