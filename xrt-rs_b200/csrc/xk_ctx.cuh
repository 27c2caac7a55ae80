// The context object behind the opaque xk_ctx handle (include/xk.h).
#pragma once

#include <string>
#include <vector>

#include "xk_internal.cuh"
#include "xk_pr.cuh"

struct xk_ctx {
    int device = 0;
    int num_sms = 0;
    bool is_shared = false;
    std::string name;
    std::string last_error;
    std::mutex mu;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    xk::F64Workspace f64ws;
    xk::PrWorkspace prws;
    xk::PrOptions pr_opts;    // .tune points at `tune`
    xk::PrTuneCache tune;     // autotuned settings per bucket of solves
    double last_energy_ev = 0.0, last_dist_mm = 0.0;  // of the last planned F32PR solve
    xk::DevBuf in_rays, in_pix, out_field;
    xk::DevBuf in_beam;  // beam columns, normals and good indices (xk_beam_* calls)
    xk::FresnelWorkspace fresnel;
    // Pinned staging of small host arrays (stage_in, stage_out).
    xk::HostBuf stage_up, stage_down;
    struct Pending {
        double* dst;
        size_t at, n;  // doubles
    };
    std::vector<Pending> pending;
};

namespace xk {

// Host arrays of up to kStageBytes per direction and call pass through pinned
// staging: one copy of all columns instead of one per column, each of which the
// driver would stage and wait for by itself (15 columns of 80 KB took 110 us).
// Arrays that are pinned already, or larger, are copied directly.
constexpr size_t kStageBytes = (size_t)2 << 20;

// `cols` host arrays of n doubles -> consecutive device columns at `dst`, through
// the staging area from double `at` on.
Status stage_in(xk_ctx* ctx, const double* const* src, int cols, double* dst, size_t n, size_t at,
                cudaStream_t s);
// Consecutive device columns at `src` -> `cols` host arrays of n doubles.
// Staged ones reach the caller's arrays in unstage().
Status stage_out(xk_ctx* ctx, double* const* dst, int cols, const double* src, size_t n, size_t at,
                 cudaStream_t s);
// After the stream is synchronised.
void unstage(xk_ctx* ctx);

}  // namespace xk
