// stt_ctx.h -- the context behind the opaque stt_ctx handle of include/stt.h
// (private to libstt.so: stt_capi.cu owns it; the solver reads its launch
// choices; the autotuner stt_tune.cu sets them and rewrites the view table).
#pragma once

#include <string>
#include <vector>

#include "stt.h"
#include "stt_internal.cuh"
#include "stt_kernels.h"

struct stt_ctx {
    int device = 0;
    std::string err;
    bool has_geom = false;
    stt::GeomDev g{};
    double sp[3] = {1, 1, 1};
    stt_geometry geom{};              // the last geometry set (its angles pointer is not kept)
    std::vector<stt::ViewRec> views_h;
    std::vector<float> off_axis_deg;  // per view: angle of the central ray off the nearest of x and z
    stt::ViewRec *views_d = nullptr;
    size_t views_cap = 0;
    float2 *acc = nullptr;  // ray-BP accumulators (contrib, weight) per voxel
    size_t acc_n = 0;
    float *corr = nullptr;  // W*H correction image used by stt_sart_sweep
    size_t corr_n = 0;
    float *volt = nullptr;  // z-fastest copy of the volume for views gathering along x
    size_t volt_n = 0;
    unsigned short *volt16 = nullptr;  // the same for a BF16-stored volume
    size_t volt16_n = 0;
    float *pw = nullptr;  // power iteration: x, A^T A x, and a chunk of projections
    size_t pw_n = 0;
    double *pwd = nullptr;  // power iteration: FP64 sums
    size_t pwd_n = 0;
    int *status = nullptr;  // raised by a bounded device-side wait that gave up (stt_poll_status)
    size_t status_n = 0;
    // Launch choices (stt_autotune / stt_set_tuning).  staged_bins: bit b set =
    // views 5b..5b+5 degrees off the nearest axis use the slab-staged projector
    // (0x1E0, 25-45 degrees, is the rule build_view applies by default).
    stt::Tuning tuning{};
    unsigned staged_bins = 0x1E0u;
    unsigned staged_bins16 = 0x1E0u;  // the same for a BF16-stored volume (ViewRec::staged16)
    // The projector's default choices: texture gathers of every view where a
    // volume of this size can bind (itself or through a mirror), and loads with the
    // oblique views staged where the one at hand does not.  Also what
    // stt_set_tuning keeps when it is given the pair that default_fp reports.
    bool fp_default = true, fp16_default = true;
    bool tex_admits = false, tex_admits16 = false;
    bool tuned = false;
    stt_tuning report{};
    // Texture objects of the tld4 gather forms for the arrays the entry points
    // were given, keyed by the array and the dimensions: at most kFpTexCache, past
    // which the older half goes (cached_tex), but those that a stream capture bound,
    // which stay valid until stt_destroy.
    struct FpTexEntry {
        const void *vol;
        int nx, ny, nz, esize;
        stt::FpTex tex;
        bool captured;
    };
    static constexpr int kFpTexCache = 256;
    std::vector<FpTexEntry> fp_tex;
    // The mirror of a volume no texture binds (launch_mirror), by storage:
    // [0] FP32, [1] BF16.  Written anew by every call that projects from it, on
    // whatever stream, so a call first waits for `read`, recorded behind the last
    // reader of the call before (as an external event in a stream capture, so a
    // replay takes its place in the order).  One that a capture uses is kept until
    // stt_destroy (`retired`), for the replays.
    struct Mirror {
        void *p = nullptr;
        cudaEvent_t read = nullptr;
        bool captured = false;
        size_t bytes = 0;
        int nx = 0, ny = 0, nz = 0;
        stt::FpTex tex;
    } mirror[2];
    std::vector<Mirror> retired;
};

namespace stt {
// Off-axis class of a view: 0..8, 5-degree classes (40-45 degrees in 8).
inline int off_axis_bin(float deg) {
    int b = (int)(deg / 5.0f);
    return b < 0 ? 0 : (b > 8 ? 8 : b);
}
// Applies ctx->staged_bins and staged_bins16 to every view (host and device tables).
stt_status apply_staged_bins(stt_ctx *ctx);
// Whether `s` is being captured: then nothing is allocated or created for it, and
// the call takes the form that needs neither.
bool capturing(cudaStream_t s);
// The texture of `vol` (created on first use, cached in the context), whatever
// the tuned variant; nullptr where it does not bind, it would have to be created
// while `s` is being captured, or captures hold the whole cache.  Valid until the
// next call.
const FpTex *ctx_fp_tex(stt_ctx *ctx, const float *vol, cudaStream_t s);
const FpTex *ctx_fp_tex(stt_ctx *ctx, const unsigned short *vol, cudaStream_t s);
// The texture of the context's mirror for volumes of this storage, and the
// mirror (allocated on first use; nullptr as above, or without memory), which `s`
// may write from here on.  The caller ends its use with ctx_mirror_done once its
// last reader is enqueued.
const FpTex *ctx_mirror_tex(stt_ctx *ctx, cudaStream_t s, float **mirror);
const FpTex *ctx_mirror_tex(stt_ctx *ctx, cudaStream_t s, unsigned short **mirror);
void ctx_mirror_done(stt_ctx *ctx, size_t esize, cudaStream_t s);
// The default pair of gather variant and staged classes, as it is reported.
struct FpDefault {
    int variant;
    unsigned staged_bins;
};
inline FpDefault default_fp(const stt_ctx *c) {
    return c->tex_admits ? FpDefault{FP_DEFAULT_TEX, 0u} : FpDefault{FP_DEFAULT_LOADS, 0x1E0u};
}
inline FpDefault default_fp16(const stt_ctx *c) { return c->tex_admits16 ? FpDefault{1, 0u} : FpDefault{0, 0x1E0u}; }
// How the correction projector runs on volumes of one storage: the choices set; by
// default tld4 corners and no view staged where the textures bind (FP_DEFAULT_TEX),
// else loads (FP_DEFAULT_LOADS; BF16 form 0) with the oblique views staged.
struct FpChoice {
    int variant;  // launch_fp_corr's fp_variant (FP32) or fp_variant16 (BF16)
    bool tex;     // its corners come from the volume's texture
    // Some view class goes to the slab-staged projector, by ViewRec::layout (its boxes
    // cover the volume for layout 0, and the z-fastest copy too for layout 1).
    bool stage[2];
};
FpChoice fp_choice(const stt_ctx *ctx, const float *, bool tex_binds);
FpChoice fp_choice(const stt_ctx *ctx, const unsigned short *, bool tex_binds);
// Whether a view gathers from the z-fastest copy under that choice.
inline bool fp_needs_copy(const FpChoice &c, const ViewRec &v, bool staged) {
    return v.layout == 1 && (!c.tex || (c.stage[1] && staged));
}
}  // namespace stt
