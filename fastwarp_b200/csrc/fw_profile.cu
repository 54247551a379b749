// fw_profile.cu -- device timing of a SyN iteration's steps with CUDA events on the context's stream
// (the timestamp profiler of the wgpu engine, crates/fastwarp-gpu/src/profiler.rs:8-60, for the
// kernels that one iteration launches at a given level grid).
#include <cuda_runtime.h>

#include <algorithm>

#include <cstring>

#include "fw_internal.cuh"

namespace fw {
namespace {

struct Events {
    cudaEvent_t a = nullptr, b = nullptr;
    ~Events() {
        if (a) cudaEventDestroy(a);
        if (b) cudaEventDestroy(b);
    }
};

}  // namespace
}  // namespace fw

using namespace fw;

extern "C" {

/* Times `reps` back-to-back runs of each step of an unmasked SyN iteration on the grid of `fixed`
 * (fixed and moving on one grid), both sides and by the kernels that the iteration launches
 * (enqueue_iteration: pair kernels, or one side after the other where two fields do not fit L2), and
 * writes the mean milliseconds and the algorithmic bytes of
 *   [0] the two warps (field + source gather + output), [1] the CC pair (2 images in, 2 fields out),
 *   [2] the Gaussian smoothing of both gradients with the max norms, [3] both compose+scale in place,
 *   [4] one inversion body of both sides as the loop runs it (its bound, step and fix kernels, after
 *   the loop's init), [5] the bound kernel alone, [6] the fix kernel alone (the tiles the step
 *   deferred; bytes counts their voxels). */
int fw_time_kernels(fw_ctx* ctx, const fw_image* fixed, const fw_image* moving, int32_t radius,
                    double variance, int32_t reps, double ms[7], double bytes[7]) {
    FW_CHECK(ctx && fixed && moving && ms && bytes && reps > 0, "null argument");
    FW_CHECK(fixed->grid.same(moving->grid), "time kernels: the images are not on one grid");
    const HostGrid& g = fixed->grid;
    const double n = (double)g.count();
    // per side: the CC derivative, the smoothed update, the inverse (and composition target), the
    // smoothing's temporary and inversion's residual
    fw_field *d[2] = {nullptr, nullptr}, *u[2] = {nullptr, nullptr}, *w[2] = {nullptr, nullptr},
             *e[2] = {nullptr, nullptr};
    fw_image* out[2] = {nullptr, nullptr};
    InvState* st = nullptr;  // the loop states: side s's at st[2 s]
    constexpr size_t st_bytes = 4 * sizeof(InvState);
    fw_grid cg = to_c(g);
    int rc = 0;
    for (int s = 0; s < 2 && !rc; ++s)
        for (fw_field** f : {&d[s], &u[s], &w[s], &e[s]})
            if (!rc) rc = fw_field_zero(ctx, &cg, f);
    for (int s = 0; s < 2 && !rc; ++s) rc = new_image(ctx, g, &out[s]);
    if (!rc) rc = dev_alloc(ctx, st_bytes, (void**)&st);
    if (!rc)  // before the slots' places in it are taken
        rc = ensure_scratch(ctx, std::max<size_t>(SLOT_PARTIALS + (size_t)(1 << 20),
                                                  inv_scratch_doubles(g)));
    Events ev;
    if (!rc && (cudaEventCreate(&ev.a) != cudaSuccess || cudaEventCreate(&ev.b) != cudaSuccess))
        rc = fail(FW_ERR_CUDA, "event creation failed");
    unsigned int* bits = ctx->d_counter + 40;
    // smooth nonzero fields for the gathers: the CC derivatives of the pair, smoothed
    if (!rc)
        rc = launch_cc_pair_impl(ctx, fixed, moving, radius, d[0], d[1],
                                 ctx->d_scratch + SLOT_CC_VALUE, 0);
    for (int s = 0; s < 2 && !rc; ++s) rc = launch_smooth(ctx, d[s], u[s], variance, bits + s, e[s]);
    if (!rc) rc = sync(ctx);
    // kinds 0-6 as documented; kind 4 includes the loops' init kernel, timed alone as kind 7 and
    // subtracted
    double t_init = 0.0;
    double deferred = 0.0;  // fraction of the step's tiles left to the fix kernel
    const fw_invert_params once = {1, -1.0, -1.0, 1};
    const int sides = syn_sides_together(g);
    const fw_image* const src[2] = {fixed, moving};
    const fw_affine* const affine[2] = {nullptr, nullptr};
    float* const warped[2] = {rc ? nullptr : out[0]->d, rc ? nullptr : out[1]->d};
    auto body = [&](int which) {
        return enqueue_inversion_pair_body(ctx, u, w, e, st, 0, 0, which);
    };
    auto zero_inverses = [&]() -> int {  // every timed body starts from psi = 0
        for (int s = 0; s < 2; ++s) FW_CUDA(cudaMemsetAsync(w[s]->d, 0, w[s]->bytes, ctx->stream));
        return 0;
    };
    for (int kind = 0; kind < 8 && !rc; ++kind) {
        auto launch = [&]() -> int {
            switch (kind) {
                case 0: return launch_warp_pair(ctx, src, u, affine, warped);
                case 1: return launch_cc_pair_impl(ctx, fixed, moving, radius, d[0], d[1],
                                                   ctx->d_scratch + SLOT_CC_VALUE, 0);
                case 2: {
                    bool in_tmp = false;
                    for (int s = 0; s < 2; s += sides)
                        FW_TRY(launch_smooth_sides(ctx, d + s, e + s, sides, variance, bits + s, &in_tmp));
                    return 0;
                }
                case 3:
                    if (sides == 2) return launch_compose_pair(ctx, u, w, bits, 0.1);
                    for (int s = 0; s < 2; ++s)
                        FW_TRY(launch_compose(ctx, u[s], w[s], w[s], bits + s, 0.1));
                    return 0;
                case 4:  // a first body of fresh loops
                    FW_TRY(enqueue_inversion_pair_init(ctx, once, st));
                    return body(-1);
                case 5: return body(0);
                case 6: return body(2);
                default: return enqueue_inversion_pair_init(ctx, once, st);
            }
        };
        if (kind == 4 || kind == 5 || kind == 6) rc = zero_inverses();
        if (!rc && (kind == 5 || kind == 6)) {  // loops before their first body (and after its step)
            rc = enqueue_inversion_pair_init(ctx, once, st);
            if (!rc && kind == 6) rc = body(0);
            if (!rc && kind == 6) rc = body(1);
        }
        if (!rc) rc = launch();  // warm-up
        if (rc) break;
        if (kind == 6) {  // the step's deferred tiles, for the fix kernel's bytes
            InvState h[3];
            double hv[sizeof(h) / sizeof(double)];
            rc = read_back(ctx, reinterpret_cast<const double*>(st), (int)(sizeof(h) / sizeof(double)), hv);
            if (rc) break;
            std::memcpy(h, hv, sizeof(h));
            deferred = (double)(h[0].ndefer + h[2].ndefer) / (2.0 * (double)inv_step_parts(g));
        }
        cudaEventRecord(ev.a, ctx->stream);
        for (int r = 0; r < reps && !rc; ++r) rc = launch();
        cudaEventRecord(ev.b, ctx->stream);
        if (rc) break;
        rc = sync(ctx);
        float t = 0.0f;
        cudaEventElapsedTime(&t, ev.a, ev.b);
        if (kind < 7) ms[kind] = (double)t / reps;
        else t_init = (double)t / reps;
    }
    if (!rc) ms[4] = std::max(ms[4] - t_init, 1e-6);
    // algorithmic bytes of the two sides: float32 voxels and field components
    bytes[0] = 2 * n * (12.0 + 4.0 + 4.0);     // field, source gather (one value), output
    bytes[1] = n * (8.0 + 24.0);               // two images in, two fields out
    bytes[2] = 2 * n * (12.0 + 12.0);          // field in, field out
    bytes[3] = 2 * n * (12.0 + 12.0 + 12.0);   // update gather, field in, field out
    bytes[4] = 2 * n * (12.0 + 12.0 + 12.0);   // psi in, field gather, psi out
    bytes[5] = 2 * (double)inv_bound_voxels(g) * 24.0;  // psi and the field gather on the lattice
    bytes[6] = 2 * deferred * n * 36.0;        // psi and residual in, psi out, deferred voxels
    for (int s = 0; s < 2; ++s) {
        for (fw_field* f : {d[s], u[s], w[s], e[s]}) fw_field_free(f);
        fw_image_free(out[s]);
    }
    if (st) dev_free(ctx, st, st_bytes);
    return rc;
}

}  // extern "C"
