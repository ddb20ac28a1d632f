// Mixed-precision regular-box right-hand side (OCFD_FLUX_FP32): the kernel of
// rhs_regular_kernel.cuh instantiated with FP32 primitives, split, WENO-Z,
// viscous flux and divergence; FP64 state and RK accumulation.
#include <cuda_runtime.h>

#include "rhs_regular_kernel.cuh"

namespace ocfd {

ocfd_status configure_rhs_regular_f32() { return configure_all<float>(); }

ocfd_status launch_rhs_regular_f32(int tile, bool visc, const RegBoxArgs* d_boxes,
                               const int* d_tile_start, int nbox, const RegBoxArgs& single,
                               int ntiles, const DevParm& P, cudaStream_t st, int sched, unsigned* queue) {
    return launch_any<float>(tile, visc, d_boxes, d_tile_start, nbox, single, ntiles, P, st, sched, queue);
}

static ocfd_status box_f32(int tile, int32_t* staged, ocfd_context* ctx, const ocfd_array4* S, const ocfd_array4* dSdt,
                           const ocfd_array4* flux, const ocfd_box& bx, const double dxinv[3], unsigned flags,
                           void* stream) {
    RegBoxArgs a{};
    fill_regular_args(a, S, dSdt, flux, bx, dxinv, tile);
    if (staged) *staged = a.use_tma;
    const int ntiles = a.ntile[0] * a.ntile[1] * a.ntile[2];
    DevParm P = ctx->parm;
    P.grav = (flags & OCFD_GRAVITY) ? kGravity : 0.0;
    return launch_any<float>(tile, (flags & OCFD_VISC) != 0, nullptr, nullptr, 1, a, ntiles, P,
                             static_cast<cudaStream_t>(stream));
}

ocfd_status rhs_regular_box_f32(ocfd_context* ctx, const ocfd_array4* S, const ocfd_array4* dSdt,
                                const ocfd_array4* flux, const ocfd_box& bx,
                                const double dxinv[3], unsigned flags, void* stream) {
    const int n[3] = {bx.hi[0] - bx.lo[0] + 1, bx.hi[1] - bx.lo[1] + 1, bx.hi[2] - bx.lo[2] + 1};
    const int tile = pick_regular_tile(n, (flags & OCFD_VISC) != 0, true, ctx->num_sms);
    return box_f32(tile, nullptr, ctx, S, dSdt, flux, bx, dxinv, flags, stream);
}

}  // namespace ocfd

extern "C" ocfd_status ocfd_check_rhs_f32_tile(ocfd_context* ctx, const ocfd_array4* S, const ocfd_array4* dSdt,
                                               const ocfd_array4* flux, ocfd_box bx, const double dxinv[3], int32_t tile,
                                               int32_t* staged, void* stream) {
    using namespace ocfd;
    if (!ctx || !dxinv || !flux || !staged || tile < 0 || tile >= kNumPublicTiles || !covers(S, bx, 3, 5) ||
        !covers(dSdt, bx, 0, 5))
        return fail(OCFD_BAD_ARG, "ocfd_check_rhs_f32_tile");
    for (int d = 0; d < 3; ++d)
        if (bx.hi[d] < bx.lo[d] || !covers(&flux[d], bx, 0, 5, d)) return fail(OCFD_BAD_ARG, "ocfd_check_rhs_f32_tile");
    return box_f32(tile, staged, ctx, S, dSdt, flux, bx, dxinv, 0, stream);
}
