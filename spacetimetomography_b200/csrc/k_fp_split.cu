// k_fp_split.cu -- the forward projector for views with few rays: P warps of a
// block share one tile of 32 rays.
//
// A view of 128^2 has 512 warps of rays, 3.5 per SM, each a chain of some 20
// rounds of gathers: the latency of those rounds is its time.  With 4 warps a ray
// the chain is a quarter as long.  Per view, us, views at 0 / 45 / 90 degrees,
// one thread a ray (gather variant 10) -> this: 64^3 / 96^2 15/14/14 -> 10/11/10,
// 96^3 / 128^2 17/17/15 -> 13/12/13, 128^3 / 128^2 17/21/17 -> 15/14/15; past
// about 24,000 rays the ray set-up and steps that every warp repeats cost more
// than the latency saved (128^3 / 192^2 19/23/19 -> 22/22/22, 256^3 / 512^2
// 119/122/116 -> 164/163/160), so there the one-thread form stays.  Measured and
// not kept: 8 warps a ray (20 to 25 at 128^3), 8 samples each in flight (151
// registers: 16), tiles of 32 x 1 (16/18/16).
#include "stt_internal.cuh"
#include "stt_kernels.h"

namespace stt {

namespace {

// The ray sums of a block's 32 rays (one per lane), by P warps: every warp
// replays the march of all 32 rays (the same float additions, so the same
// positions), and in a round of P*G samples warp `part` fetches and
// interpolates samples part*G .. part*G + G - 1.  The products go to shared
// memory; warp 0 adds them in march order to the compensated sum while the
// others start the next round.  So the samples, their roundings and their
// order are those of fp_ray_sum_with, with P*G of them in flight per ray
// instead of G.  Every thread of the block calls this (one barrier per round).
// The result and the sample count are warp 0's.
template <int P, int G, typename Corners>
__device__ __forceinline__ float fp_ray_sum_split(const GeomDev &g, const Corners &corners, const Ray &r, bool hit,
                                                  int part, int lane, float (*vals)[P * G][32], int &count) {
    constexpr int S = P * G;
    static_assert(G % 2 == 0, "samples go in packed pairs");
    Kahan acc{0.0f, 0.0f};
    count = 0;
    const float sd = g.sd, tnear = r.tnear, tfar = r.tfar;
    MarchDda d;
    float pos1[3], t1 = tnear, t = 0.0f, tb = 0.0f;
    float2 xy = f2(0.0f, 0.0f), tz = f2(0.0f, 0.0f);  // the round's first sample: (x, y), (t, z)
    int seg = -1, n = 0, cap = 0, budget = 1 << 22;
#pragma unroll
    for (int k = 0; k < 3; ++k) pos1[k] = __fadd_rn(r.vz[k], __fmul_rn(r.vu[k], tnear));
    if (hit) march_dda(g, r, pos1, d);
    // the next segment that holds a sample; false when the ray is done
    auto next_segment = [&]() -> bool {
        while (true) {
            if (seg >= 0) {
                march_split(d);
                t1 = tb;
            }
            if (!(++seg < 16 && t1 < tfar && budget > 0)) return false;
            tb = rmin(rmin(d.tmax[0], d.tmax[1]), d.tmax[2]);
            if (tb > tfar) tb = tfar;
            t = __fadd_rn(__fmul_rn(ceilf(__fdiv_rn(__fsub_rn(t1, tnear), sd)), sd), tnear);
            xy = f2(__fadd_rn(r.vz[0], __fmul_rn(r.vu[0], t)), __fadd_rn(r.vz[1], __fmul_rn(r.vu[1], t)));
            tz = f2(t, __fadd_rn(r.vz[2], __fmul_rn(r.vu[2], t)));
            cap = (int)fminf(ceilf(__fdiv_rn(tb - t, sd)) + 2.0f, (float)budget);
            budget -= cap > 0 ? cap : 0;
            n = 0;
            if (n < cap && t < tb) return true;
        }
    };
    bool live = hit && next_segment();
    if (hit && part == 0) {
        // The entry sample.  The first segment usually starts on it (t = tnear):
        // then its product is the first one of the round, added twice.
        if (!(live && seg == 0)) {
            FpCell c;
            fp_cell(g, pos1, c);
            float v[8];
            corners(0, c, v);
            acc.add(__fmul_rn(trilerp(v, c), sd));
        }
        ++count;
    }
    bool twice = live && seg == 0;
    int buf = 0;
    // One barrier a round: a buffer is written again two rounds on, after a
    // barrier that warp 0 reaches only when it has read it.
    for (bool more = __syncthreads_or(live); more; buf ^= 1) {
        int have = 0;  // samples of this round
        if (live) {
            const float2 sxy = f2(d.step[0], d.step[1]), stz = f2(sd, d.step[2]);
            float2 axy = xy, atz = tz;
#pragma unroll
            for (int q = 0; q < P - 1; ++q)
                if (q < part)
#pragma unroll
                    for (int i = 0; i < G; ++i) axy = __fadd2_rn(axy, sxy), atz = __fadd2_rn(atz, stz);
            FpCell c[G];
            float v[G][8];
#pragma unroll
            for (int i = 0; i < G; i += 2) {
                const float2 bxy = __fadd2_rn(axy, sxy), btz = __fadd2_rn(atz, stz);
                const float pa[3] = {axy.x, axy.y, atz.y}, pb[3] = {bxy.x, bxy.y, btz.y};
                fp_cell2(g, pa, pb, c[i], c[i + 1]);
                corners(i, c[i], v[i]);
                corners(i + 1, c[i + 1], v[i + 1]);
                axy = __fadd2_rn(bxy, sxy), atz = __fadd2_rn(btz, stz);
            }
            // the rest of the round's steps, to the next round's first sample
#pragma unroll
            for (int q = 1; q < P; ++q)
                if (q > part)
#pragma unroll
                    for (int i = 0; i < G; ++i) axy = __fadd2_rn(axy, sxy), atz = __fadd2_rn(atz, stz);
            const float2 sd2 = f2(sd, sd);
#pragma unroll
            for (int i = 0; i < G; i += 2) {
                const float2 s = __fmul2_rn(trilerp2(v[i], v[i + 1], c[i], c[i + 1]), sd2);
                vals[buf][part * G + i][lane] = s.x;
                vals[buf][part * G + i + 1][lane] = s.y;
            }
            // how many of the round's samples the segment holds (t only grows)
            if (n + S <= cap && atz.x < tb) {
                have = S;
            } else {
                float tt = tz.x;
                while (have < S && n + have < cap && tt < tb) ++have, tt = __fadd_rn(tt, sd);
            }
            xy = axy, tz = atz;
            n += S;
            if (have < S || !(n < cap && tz.x < tb)) live = next_segment();
        }
        more = __syncthreads_or(live);
        if (part == 0 && have > 0) {
            if (twice) acc.add(vals[buf][0][lane]);
            twice = false;
            if (have == S) {
#pragma unroll
                for (int i = 0; i < S; ++i) acc.add(vals[buf][i][lane]);
            } else {
                for (int i = 0; i < have; ++i) acc.add(vals[buf][i][lane]);
            }
            count += have;
        }
    }
    return acc.s;
}

// What a projection writes for its rays: the projection of views
// [view0, view0 + gridDim.z) (k_fp's outputs), or one view's correction
// (k_fp_corr's).
struct ProjOut {
    int view0;
    float *proj, *raylen, *weight;
    __device__ __forceinline__ int view() const { return view0 + blockIdx.z; }
    __device__ __forceinline__ void write(const GeomDev &g, size_t pix, bool hit, float len, float sum, int count) const {
        const size_t o = (size_t)blockIdx.z * g.W * g.H + pix;
        proj[o] = sum;
        if (raylen && hit) raylen[o] = len;
        if (weight) weight[o] = (float)count;
    }
};
template <typename B>
struct CorrOut {
    ViewSel sel;
    const B *b_stack;
    float *raylen_state, *corr;
    __device__ __forceinline__ int view() const {
        int local;
        return sel_view(sel, local);
    }
    __device__ __forceinline__ void write(const GeomDev &g, size_t pix, bool hit, float len, float sum, int) const {
        int local;
        sel_view(sel, local);
        float L;
        if (hit) {
            L = len;
            if (raylen_state) raylen_state[pix] = L;
        } else {
            L = raylen_state ? raylen_state[pix] : 0.0f;
        }
        const float b = ld_voxel(b_stack + (size_t)local * g.W * g.H + pix);
        corr[pix] = __fdiv_rn(__fsub_rn(b, sum), __fadd_rn(L, 1.0f));
    }
};

// A block is 8 x 4 pixels; T: the volume's storage.
constexpr int SPLIT_P = 4, SPLIT_G = 4;
template <typename T, typename Out>
__global__ void __launch_bounds__(32 * SPLIT_P) k_fp_split(const GeomDev g, const ViewRec *__restrict__ views,
                                                           const Out out, const FpTex tex, int skip_staged) {
    __shared__ float vals[2][SPLIT_P * SPLIT_G][32];
    const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
    const int i = blockIdx.x * 8 + (lane & 7), j = blockIdx.y * 4 + (lane >> 3);
    const bool pixel = i < g.W && j < g.H;
    const ViewRec &vr = views[out.view()];
    if (skip_staged && view_staged<T>(vr)) return;  // the slab-staged kernel projects this view
    Ray r;
    make_ray(g, vr, min(i, g.W - 1), min(j, g.H - 1), r);
    const bool hit = pixel && r.tnear < r.tfar;
    const unsigned long long t = tex.x;
    const int nx = g.nx;
    int count;
    const float sum = fp_ray_sum_split<SPLIT_P, SPLIT_G>(
        g, [=](int, const FpCell &c, float w[8]) { fp_corners_tex<T>(t, nx, c, w); }, r, hit, part, lane, vals, count);
    cudaTriggerProgrammaticLaunchCompletion();
    if (part == 0 && pixel) out.write(g, i + (size_t)j * g.W, hit, r.tfar - r.tnear, sum, count);
}

template <typename T, typename Out>
cudaError_t split(const GeomDev &g, const ViewRec *views, const Out &out, int nviews, cudaStream_t s, const FpTex &tex,
                  int skip_staged) {
    k_fp_split<T><<<dim3((g.W + 7) / 8, (g.H + 3) / 4, nviews), 32 * SPLIT_P, 0, s>>>(g, views, out, tex, skip_staged);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_fp_split(const GeomDev &g, const ViewRec *views, int view0, int nviews, float *proj, float *raylen,
                            float *weight, cudaStream_t s, const FpTex &tex) {
    const ProjOut out{view0, proj, raylen, weight};
    return tex.esize == 2 ? split<unsigned short>(g, views, out, nviews, s, tex, 0)
                          : split<float>(g, views, out, nviews, s, tex, 0);
}

cudaError_t launch_fp_corr_split(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *b_stack,
                                 float *raylen_state, float *corr, cudaStream_t s, const FpTex &tex, int skip_staged) {
    return split<float>(g, views, CorrOut<float>{sel, b_stack, raylen_state, corr}, 1, s, tex, skip_staged);
}

cudaError_t launch_fp_corr_split(const GeomDev &g, const ViewRec *views, const ViewSel &sel,
                                 const unsigned short *b_stack, float *raylen_state, float *corr, cudaStream_t s,
                                 const FpTex &tex, int skip_staged) {
    return split<unsigned short>(g, views, CorrOut<unsigned short>{sel, b_stack, raylen_state, corr}, 1, s, tex,
                                 skip_staged);
}

}  // namespace stt
