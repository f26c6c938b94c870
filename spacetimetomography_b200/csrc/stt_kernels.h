// stt_kernels.h -- host-side launch wrappers of the kernels in k_*.cu.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

namespace stt {

struct ViewRec;
struct GeomDev;
struct ViewSel;

struct PdParams {
    float sigma, tau, tv_w, tp_w, bc_w, hf, gmax;
    int cut[8];
};

// A launch that may start before the kernel ahead of it in the stream has
// finished: its blocks take the places that kernel's last blocks leave, and wait
// in cudaGridDependencySynchronize(), which the kernel calls before it touches
// anything another kernel writes or reads, until it has.  What that kernel writes is
// read after the wait and not through the read-only or texture path, whose data may
// not change while a grid runs.  A kernel that calls
// cudaTriggerProgrammaticLaunchCompletion() lets its successor come up early.
template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, cudaStream_t s, Args &&...args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// Multiprocessor count of the current device (cached per device).
int sm_count();
int grid_stride_blocks(long long n, int threads);

// Launch shapes of the tunable kernels, picked by the autotuner (stt_tune.cu).
// Variant 0 of each is the default; all variants of a kernel give the same
// bits (they change which thread or block computes what, never a value's
// arithmetic).
//   fp:   the gather forward projector k_fp_corr: detector tile, samples
//         in flight and, for variants 10 and 11, corners fetched as two tld4
//         texture gathers per sample instead of eight loads (fp_variant_name);
//   slab: the box of the slab-staged projector (slab_variant_name);
//   bp:   the column length of the voxel backprojection and the blocks per SM
//         it is compiled for (bp_variant_name);
//   ray:  the scatter of the ray-driven backprojection (ray_variant_name):
//         0 global vector atomics, neighbouring rows merged, 1 a shared-memory
//         box per slab (volumes below 2^31 voxels).  Its sums differ in float order
//         only (as any two atomic runs do), not in their terms.
// Which views the slab kernel projects is the per-view ViewRec::staged flag.
constexpr int kFpVariants = 12, kSlabVariants = 8, kBpVariants = 5, kRayVariants = 2;
struct Tuning {
    int fp = 0, slab = 0, bp = 0, ray = 0;
    int fp16 = 0;  // the BF16-stored volume's gather form (fp16_variant_name)
};
const char *fp_variant_name(int v);
const char *slab_variant_name(int v);
const char *bp_variant_name(int v);
const char *ray_variant_name(int v);
// The scatter an untuned context uses (k_scatter.cu has the measurements).
int default_ray_variant(const GeomDev &g);

// The projection of nviews views: corners through the textures of `tex` where
// it is usable (the same values), else by loads from vol, or from vol_t for
// the views along x when it is given.
struct FpTex;
cudaError_t launch_fp(const GeomDev &g, const ViewRec *views, const float *vol, const float *vol_t, int view0,
                      int nviews, float *proj, float *raylen, float *weight, cudaStream_t s,
                      const FpTex *tex = nullptr);
// Slab-staged forward projector (k_fp_slab.cu) for the views marked `staged`:
// the same outputs as the gather form bit for bit, the volume read through
// TMA boxes.  The tensor maps cover the volume and its z-fastest copy (vol_t
// may be null: then every view gathers from vol) with the box of slab variant
// `variant`; make_fp_slab_maps returns false where the form does not apply (x
// or z extent not a multiple of 4, an array not 16-byte aligned, 2^31 voxels
// or more).  `status` (may be null) is set to 1 if a box copy did not land
// within the wait limit.
struct FpSlabMaps {
    CUtensorMap x, z;
    int ok, has_z, variant;
    int esize;  // bytes per voxel: 4 (FP32) or 2 (BF16)
};
bool make_fp_slab_maps(const GeomDev &g, const float *vol, const float *vol_t, FpSlabMaps &m, int variant = 0);
// BF16 storage: the scalar boxes (variant & 3); x and z extents multiples of 8.
bool make_fp_slab_maps(const GeomDev &g, const unsigned short *vol, const unsigned short *vol_t, FpSlabMaps &m,
                       int variant = 0);
// Whether the maps' extents admit volumes of this size (esize bytes per voxel), and
// with `copy` their z-fastest copies too.
bool fp_slab_fits(const GeomDev &g, int esize, bool copy);
// A 4D FP32 tensor map over nc planar volumes (x fastest, then y, z, plane)
// with the given box (x, y, z, plane); false where TMA cannot address them
// (nx not a multiple of 4, ptr not 16-byte aligned, box row not 16 bytes).
bool encode_planes_map(CUtensorMap *m, const float *ptr, int nx, int ny, int nz, int nc, const unsigned box[4]);
cudaError_t launch_fp_corr_slab(const GeomDev &g, const ViewRec *views, const FpSlabMaps &m, const float *vol,
                                const float *vol_t, const ViewSel &sel, const float *b_stack, float *raylen_state,
                                float *corr, cudaStream_t s, int *status);
cudaError_t launch_fp_corr_slab(const GeomDev &g, const ViewRec *views, const FpSlabMaps &m,
                                const unsigned short *vol, const unsigned short *vol_t, const ViewSel &sel,
                                const unsigned short *b_stack, float *raylen_state, float *corr, cudaStream_t s,
                                int *status);
// Texture object of the gather forms that fetch corners with tld4: the volume
// as a pitch-linear 2D texture whose rows are its z slices (width nx*ny texels,
// nz rows); FP32 texels, or for a BF16-stored volume 16-bit unsigned texels
// holding its bits.  Point sampling returns stored values exactly, so the
// samples are those of the loads they replace.  A gather's footprint is two
// texels of two slices whatever the ray's direction, so every view reads the
// volume itself: no z-fastest copy.  make_fp_tex returns false (and creates
// nothing) where the device's limits on linear 2D textures do not admit the
// array: a row of more than the maximum width or pitch, more rows than the
// maximum height, a base not aligned to the texture alignment.  The caller owns
// the object (destroy_fp_tex).
struct FpTex {
    unsigned long long x = 0;
    int ok = 0;
    int esize = 0;  // bytes per texel: 4 (FP32) or 2 (BF16)
};
bool is_tex_fp_variant(int fp_variant);
// pitch: elements from one slice to the next (0: nx*ny).
bool make_fp_tex(const GeomDev &g, const float *vol, FpTex &t, size_t pitch = 0);
bool make_fp_tex(const GeomDev &g, const unsigned short *vol, FpTex &t, size_t pitch = 0);
// A volume whose slices the texture unit cannot step over (nx*ny not a multiple
// of the pitch alignment, an odd frame's base) is projected from a mirror: the
// same voxels with each slice starting on fp_mirror_pitch elements.  A sweep
// copies the volume there once and the voxel backprojection writes both.
// Measured against loads (with the z-fastest copy for the views along x): 15
// views of 333 x 301 of a 187 x 203 x 171 BF16 volume 531 -> 332 us, mirror
// included; a batch of eight cubes of 65 to 124 voxels 5.06 -> 3.51 ms.
inline size_t fp_mirror_pitch(size_t slice) { return (slice + 63) / 64 * 64; }
// Elements from one mirror to the next of several in one allocation (512 bytes
// at either storage, the texture base alignment).
inline size_t fp_mirror_stride(size_t slice, size_t nz) { return (fp_mirror_pitch(slice) * nz + 255) / 256 * 256; }
cudaError_t launch_mirror(const GeomDev &g, const float *vol, float *mirror, cudaStream_t s);
cudaError_t launch_mirror(const GeomDev &g, const unsigned short *vol, unsigned short *mirror, cudaStream_t s);
// Whether make_fp_tex admits `vol` (esize bytes per voxel) on this device
// (checks the limits only; creates nothing).
bool fp_tex_fits(const GeomDev &g, const void *vol, int esize, size_t pitch = 0);
// Whether one of this size can bind: at an aligned base, or its mirror.
bool fp_tex_admits(const GeomDev &g, int esize);
void destroy_fp_tex(FpTex &t);
// Projections of at most this many rays in one launch share each ray between
// the 4 warps of a block when their corners come from a texture (k_fp_split.cu).
constexpr long long FP_SPLIT_RAYS = 24576;
// Of `chains` sequences of views that run side by side (a solver's frames, a
// batch's instances) each gets a share of the GPU, which the steps that the warps
// repeat waste: eight cubes of 65 to 124 voxels, views of 80^2 to 160^2, all split
// 3.47 ms, up to 8192 rays 3.05, none 3.13; but three of 70^2 to 141^2 1.41, 1.58,
// 1.78; five of 51^2 to 102^2 0.98, 0.99, 1.14.
constexpr long long FP_SPLIT_SHARED_RAYS = 65536;
inline long long fp_split_rays(int chains) {
    const long long share = FP_SPLIT_SHARED_RAYS / (chains > 1 ? chains : 1);
    return share < FP_SPLIT_RAYS ? share : FP_SPLIT_RAYS;
}
// Where a call's projections fetch their corners: by loads; from the volume's own
// texture or, where none binds, by loads; or from a texture, of a mirror if need be.
// views[l][b]: the call's views of ViewRec::layout l in off-axis class b (5 degrees
// each); rays: of all of them; own: the volume's own texture binds.
//
// Textures are the faster by far for oblique views (the loads' lanes fall on more
// lines) and for few rays (the split form), and BF16 ones almost always.  But a copy
// of the volume costs some 0.45 us a megabyte, and along an axis loads are as fast or
// faster where FP32 volumes stay in the L2.  Loads / own texture, us, at 0 degrees,
// views x detector: 128^3 8 x 128^2 40 / 47, 24 x 64^2 37 / 48, 192^3 8 x 512^2
// 520 / 623, 256^3 8 x 512^2 730 / 852, 24 x 64^2 75 / 117 (at 20 degrees 113 / 117, at
// 45 218 / 120); but 256^3 1 x 256^2 56 / 40, 320^3 8 x 512^2 1211 / 1090.  Loads /
// mirror, one view: 255^3 512^2 at 0 degrees 106 / 144, at 20 125 / 147, at 30 163 /
// 147, 128^2 48 / 50; 187^3 128^2 37 / 27, 256^2 37 / 41; 301^3 256^2 112 / 98; a BF16
// 301^3 256^2 60 / 74, 128^2 64 / 53.
enum class FpFrom { Loads, OwnTexture, Texture };
struct FpCall {
    int views[2][9] = {};
    long long rays = 0;
};
FpFrom fp_from(long long voxels, float row_pitch, int esize, bool own, const FpCall &c);
cudaError_t launch_fp_split(const GeomDev &g, const ViewRec *views, int view0, int nviews, float *proj, float *raylen,
                            float *weight, cudaStream_t s, const FpTex &tex);
cudaError_t launch_fp_corr_split(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *b_stack,
                                 float *raylen_state, float *corr, cudaStream_t s, const FpTex &tex, int skip_staged);
cudaError_t launch_fp_corr_split(const GeomDev &g, const ViewRec *views, const ViewSel &sel,
                                 const unsigned short *b_stack, float *raylen_state, float *corr, cudaStream_t s,
                                 const FpTex &tex, int skip_staged);
// The gather form an untuned context uses where the texture binds: tld4
// corners, no view staged.  Measured against loads with the oblique views
// staged (the form before), per view, us, views at 0 / 45 / 90 degrees:
// 64^3 / 96^2 19/31/28 -> 10/11/10, 128^3 / 128^2 33/59/46 -> 15/14/15,
// 192^3 / 256^2 45/93/66 -> 31/36/30, 256^3 / 512^2 124/213/176 -> 118/122/116
// (the times before include the z-fastest copy of the views along x).
constexpr int FP_DEFAULT_TEX = 10;
// And where no texture binds (slices past the texture width): loads with two
// samples in flight.  Both forms have 64 registers, so the warps are as many; four
// samples' 32 loads a thread only lengthen the bursts that share the L1.
// Views at 0 and 90 degrees, us, four in flight -> two: 128^3 / 128^2 31/47 -> 26/37,
// 256^3 / 512^2 118/171 -> 108/160, 400^3 / 800^2 459/614 -> 406/531, 512^3 / 1024^2
// 895/1177 -> 793/1008 (the oblique views are staged, 1230); a BF16 volume's loads
// gain nothing (765/964 -> 771/953) and keep four.
constexpr int FP_DEFAULT_LOADS = 5;
// Forward projection of one view fused with the SART correction.  With usable
// slab maps, staged views run in the slab-staged kernel and the others in the
// gather kernel (both are launched; each leaves the other's views alone).
// `fp_variant` selects the gather kernel's launch shape; a texture variant
// (is_tex_fp_variant) without usable `tex` runs the load-based variant of the
// same shape, which gives the same bits.
cudaError_t launch_fp_corr(const GeomDev &g, const ViewRec *views, const float *vol, const float *vol_t,
                           const ViewSel &sel, const float *b_stack, float *raylen_state, float *corr,
                           cudaStream_t s, const FpSlabMaps *maps = nullptr,
                           int *status = nullptr, int fp_variant = 0, const FpTex *tex = nullptr,
                           int chains = 1);
cudaError_t launch_transpose(const GeomDev &g, const float *in, float *out, cudaStream_t s);
cudaError_t launch_fp(const GeomDev &g, const ViewRec *views, const unsigned short *vol, const unsigned short *vol_t,
                      int view0, int nviews, float *proj, float *raylen, float *weight, cudaStream_t s,
                      const FpTex *tex = nullptr);
cudaError_t launch_transpose_bf16(const GeomDev &g, const unsigned short *in, unsigned short *out, cudaStream_t s);
// The copy for the selected view, if it gathers from one: a view along x, and
// with staged_only (the gather form reads the volume's texture) only one that
// the slab-staged kernel projects.
cudaError_t launch_transpose_for_view(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *in,
                                      float *out, cudaStream_t s, bool staged_only = false);
cudaError_t launch_transpose_for_view(const GeomDev &g, const ViewRec *views, const ViewSel &sel,
                                      const unsigned short *in, unsigned short *out, cudaStream_t s,
                                      bool staged_only = false);

// BF16 storage (the raw upper halves of FP32 values; the solver's
// stt_solve_cfg.storage): the overloads below on unsigned short arrays read
// stored values widened exactly to FP32, compute as their FP32 forms do, and
// round what they store to nearest even.  Duals, flows, corrections and
// accumulators stay FP32.
// The fused forward projection of a BF16 volume against a BF16 sinogram:
// with usable BF16 slab maps the staged views run in the slab kernel (BF16
// boxes), the others in the gather kernel; without them every view gathers.
// The gather kernel loads its corners (fp_variant16 0: 32x4 rays, 4 samples
// in flight) or, with usable BF16 textures `tex`, gathers them with tld4
// (fp_variant16 1: warps of 8x4 rays, 8 samples in flight in packed pairs);
// the same bits either way.
constexpr int kFp16Variants = 2;
const char *fp16_variant_name(int v);
cudaError_t launch_fp_corr(const GeomDev &g, const ViewRec *views, const unsigned short *vol,
                           const unsigned short *vol_t, const ViewSel &sel, const unsigned short *b_stack,
                           float *raylen_state, float *corr, cudaStream_t s,
                           const FpSlabMaps *maps = nullptr, int *status = nullptr, int fp_variant16 = 0,
                           const FpTex *tex = nullptr, int chains = 1);
cudaError_t launch_correction(long long n, const unsigned short *b, const float *ax, const float *raylen,
                              float *corr, cudaStream_t s);
cudaError_t launch_correction(long long n, const float *b, const float *ax, const float *raylen,
                              float *corr, cudaStream_t s);
// Ray-driven backprojection: the scatter into acc (interleaved contribution,
// weight), then vol += contribution/weight and acc cleared.  The scatter is
// ray variant `ray_variant` (-1: default_ray_variant): a global atomic per
// corner, or a shared-memory box per slab (k_bp_slab.cu, below 2^31 voxels).
cudaError_t launch_bp_ray(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                          float2 *acc, float *vol, float gmax, cudaStream_t s, int ray_variant = -1);
cudaError_t launch_bp_ray(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                          float2 *acc, unsigned short *vol, float gmax, cudaStream_t s, int ray_variant = -1);
cudaError_t launch_bp_ray_scatter_slab(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                                       float2 *acc, cudaStream_t s);
cudaError_t launch_bp_ray_scatter(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                                  float2 *acc, float *contrib, float *wsum, cudaStream_t s, int ray_variant = -1);
// dense: the residual is nowhere zero.  adjoint_rays: the rays a thread it then
// marches (k_scatter.cu has the measurements).
cudaError_t launch_fp_adjoint(const GeomDev &g, const ViewRec *views, int view0, int nviews,
                              const float *proj_bar, float *vol_bar, cudaStream_t s, bool dense = false);
int adjoint_rays(const GeomDev &g, int nviews, bool dense);
// The gather ceiling (k_project.cu): one view's rays sampled at the
// projector's step with its gathers and interpolation and none of its march
// control; `host_view` is the view's record (its layout picks vol_t).  With
// `tex` (made over vol and vol_t) the corners are tld4 gathers in packed pairs.
cudaError_t launch_gather_ceiling(const GeomDev &g, const ViewRec *views, const ViewRec &host_view, int view,
                                  const float *vol, const float *vol_t, int packed, float *out, int *count,
                                  cudaStream_t s, const FpTex *tex = nullptr);
cudaError_t launch_fill_zero(float *p, long long n, cudaStream_t s);
cudaError_t launch_dot_f64(long long n, const float *a, const float *b, double *out, cudaStream_t s);
cudaError_t launch_scale_inv_sqrt(long long n, float *x, const double *norm2, cudaStream_t s);
cudaError_t launch_fill_seeded(long long n, unsigned long long seed, float *x, cudaStream_t s);

// The persistent sweep (k_persist.cu): the SART calls of all jobs (frames or
// batch instances, SweepJob in stt_internal.cuh) in one cooperative launch of
// `nblocks` blocks, jobs_d a device array sorted by block0.  bf16: the jobs'
// storage; wide: some job's volume takes 64-bit offsets (sweep_wide: 2^31 voxels or
// more, or an extent of two, whose warps only that form samples).
struct SweepJob;
bool sweep_wide(const GeomDev &g);
// Blocks of the launch that can be resident at once on the current device (0
// on error): the most a launch may have.
int sweep_max_blocks(bool bf16, bool wide);
// Orders the jobs into rounds (largest first, at most nblocks jobs a round:
// one round unless there are more jobs than blocks) and splits the nblocks
// over each round's jobs in proportion to their work: sets round, block0 and
// nblocks and sorts the array by round.  Returns the number of rounds.
int sweep_plan(SweepJob *jobs, int njobs, int nblocks);
cudaError_t launch_sweep_persistent(const SweepJob *jobs_d, int njobs, int nblocks, bool bf16, bool wide,
                                    int *status, cudaStream_t s);
// The whole primal-dual iteration of every job (view order, warps, dual and
// primal steps, then the SART call) in one cooperative launch; one round (at
// most nblocks jobs); gbar: two words zeroed before the launch, like the
// jobs' barrier words.
cudaError_t launch_iter_persistent(const SweepJob *jobs_d, int njobs, int nblocks, bool bf16, bool wide,
                                   unsigned *gbar, int *status, cudaStream_t s);

// Voxel-driven backprojection, bp variant `bp_variant` (0: columns of g.bp_len
// voxels); every voxel it writes goes to `mirror` too, if given.
// bp_default_len: the longest column whose detector rows fit in the kernel's
// table at `rows` detector rows per voxel (the geometry's largest); 8 where only
// a shorter one would and the volume is large.
int bp_default_len(double rows, long long voxels);
cudaError_t launch_bp_voxel(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                            float *vol, float alpha, float gmax, cudaStream_t s, int bp_variant = 0,
                            float *mirror = nullptr);
cudaError_t launch_bp_voxel(const GeomDev &g, const ViewRec *views, const ViewSel &sel, const float *corr,
                            unsigned short *vol, float alpha, float gmax, cudaStream_t s, int bp_variant = 0,
                            unsigned short *mirror = nullptr);
// Sets the solver's device-side iteration counter (stream-ordered, no host memory read).
cudaError_t launch_set_counter(unsigned long long *counter, unsigned long long v, cudaStream_t s);
// View orders of `frames` local frames (at most 1024), local frame f being
// frame frame0 + f of a sequence of `total`; advances *counter.
cudaError_t launch_make_perm(unsigned long long seed, unsigned long long *counter, int frames, int total,
                             int frame0, int views, int *perm, cudaStream_t s);
cudaError_t launch_pd_dual(const int *dims, const PdParams &p, const float *xf, const float *xf1,
                           const float *bw, float *ytv, float *ytp, float *ybc, cudaStream_t s);
cudaError_t launch_pd_dual(const int *dims, const PdParams &p, const unsigned short *xf, const unsigned short *xf1,
                           const float *bw, float *ytv, float *ytp, float *ybc, cudaStream_t s);
cudaError_t launch_pd_primal(const int *dims, const PdParams &p, int first, const float *ytp_prev,
                             const float *ytp, const float *fw, const float *ybc, const float *ytv,
                             float *vol, float *xprev, cudaStream_t s);
cudaError_t launch_pd_primal(const int *dims, const PdParams &p, int first, const float *ytp_prev,
                             const float *ytp, const float *fw, const float *ybc, const float *ytv,
                             unsigned short *vol, unsigned short *xprev, cudaStream_t s);
cudaError_t launch_pd_extrapolate(const int *dims, const int *cut, const float *vol,
                                  const float *xprev, float *xbar, cudaStream_t s);
cudaError_t launch_pd_extrapolate(const int *dims, const int *cut, const unsigned short *vol,
                                  const unsigned short *xprev, unsigned short *xbar, cudaStream_t s);
cudaError_t launch_roi_apply(const int *dims, const int *roi_cut, const int *pd_cut, float *vol,
                             const float *xprev, float *xbar, cudaStream_t s);
cudaError_t launch_roi_apply(const int *dims, const int *roi_cut, const int *pd_cut, unsigned short *vol,
                             const unsigned short *xprev, unsigned short *xbar, cudaStream_t s);
cudaError_t launch_roi_mask(const int *dims, const int *cut, float *roi, cudaStream_t s);

// ---- optical flow (k_flow.cu) ----
struct FlowRoi {
    int x0, x1, y0, y1, z0, z1;  // cut from each face
};

struct DericheCoef {
    float a0, a1, a2, a3, b1, b2, coefp, coefn;
};

// One axis of a CImg resize: mode 0 = moving average (shrinking), mode 1 =
// Catmull-Rom (growing) with the per-output (source index, fraction) table
// written by launch_resize_table.
struct ResizeAxis {
    int axis, mode, nc;
    int ix, iy, iz;  // input extents
    int ox, oy, oz;  // output extents (differ from the input along `axis` only)
    int old_n, new_n;
    const int *src;
    const double *frac;
};

cudaError_t launch_warp_box(const int *dim, const float *box, const float *vel, const float *src, int nc,
                            float dt, float *out, cudaStream_t s);
// The iterations' fields (float4 per voxel: v, u, steps; y packed): see Dual in
// k_flow.cu.  Y and V are the caller's planes.
cudaError_t launch_flow_pack(long long n, const float *Y, const float *V, float *y, float4 *v0, float4 *v1, float4 *v2,
                             cudaStream_t s);
cudaError_t launch_flow_setup(const int *d, const FlowRoi &roi, const float *i2w, const float *i1, const float *V,
                              float4 *u, float4 *steps, float *k4prev, cudaStream_t s);
cudaError_t launch_flow_primal(const int *d, const FlowRoi &roi, const float *y, const float4 *u, const float4 *steps,
                               const float4 *v_in, float4 *v_out, float *kty, int flags, double *resid,
                               const int *done, cudaStream_t s);
cudaError_t launch_flow_dual(const int *d, const float4 *v, const float4 *v_old, const float4 *u, const float4 *steps,
                             const float *k4prev, float *y, float sigma1, float hf, float lambda, int huber, int flags,
                             double *resid, const int *done, cudaStream_t s);
// Whether a level of that many voxels takes launch_flow_step between residual checks.
bool flow_fuses(long long voxels);
// The dual step of an iteration and the primal step of the next in one pass
// (k_flow_step); y_out and v_next are buffers of their own.
cudaError_t launch_flow_step(const int *d, const FlowRoi &roi, const float *y_in, float *y_out, const float4 *v,
                             const float4 *v_old, float4 *v_next, const float4 *u, const float4 *steps,
                             const float *k4prev, float *kty, float sigma1, float hf, float lambda, int huber,
                             int flags, const int *done, cudaStream_t s);
cudaError_t launch_flow_settle(long long n, const int *iters, const float4 *v_1, const float4 *v_2, float4 *v_0,
                               float *V, cudaStream_t s);
cudaError_t launch_flow_check(double *resid, long long n, float tol, int it, int is_resid, int is_last,
                              int *done, int *iters, float *err, cudaStream_t s);
cudaError_t launch_flow_reset(int *done, double *resid, int *iters, float *err, cudaStream_t s);
cudaError_t launch_deriche(const int *d, int nc, int axis, const DericheCoef &c, float *img, float *tmp,
                           cudaStream_t s);
cudaError_t launch_resize_table(int old_n, int new_n, int *src, double *frac, cudaStream_t s);
cudaError_t launch_resize_axis(const ResizeAxis &ra, const float *in, float *out, cudaStream_t s);
cudaError_t launch_gradient(const int *d, const float *img, float *g, cudaStream_t s);
cudaError_t launch_flow_unpack(const int *d, const FlowRoi &roi, const float *y, float *Y, cudaStream_t s);

// `status` (may be null: then a per-device word read by warp_poll_status) is
// set when the staged kernel's bounded wait for its velocity box gave up.
cudaError_t launch_warp(const int *dim, const float *vel, const float *src, int nc, float dt,
                        float *out, cudaStream_t s, int *status = nullptr);
// The warp of a BF16-stored source (taps widened to FP32; FP32 flow and output).
cudaError_t launch_warp(const int *dim, const float *vel, const unsigned short *src, int nc, float dt,
                        float *out, cudaStream_t s, int *status = nullptr);
// Reads and clears the per-device status word of warps launched without one
// (synchronises `s`); *flag is non-zero if a bounded wait gave up.
cudaError_t warp_poll_status(int *flag, cudaStream_t s);
cudaError_t launch_warp_vjp(const int *dim, const float *vel, const float *src, int nc, float dt,
                            const float *out_bar, float *src_bar, float *vel_bar, cudaStream_t s);

}  // namespace stt
