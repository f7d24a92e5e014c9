// Launch shapes of the any-shape tensor-core step, included once per precision.
#pragma once

#include "cheb_dmma_any.cuh"
#include "step_launch.cuh"

#include <type_traits>

namespace rsatb_b200 {
namespace step_detail {

template <typename VT, int B, int NG, int MT, bool CM, bool CV, bool PAIR>
int launch_dmma_any_k(rsatb_context* ctx, StepArgs& a) {
    auto kernel = cheb_step_dmma_any<VT, B, NG, MT, CM, CV, PAIR>;
    const int threads = kDmmaAnyWarps * 32;
    const int cols = CM ? a.W / 2 : a.W;
    const int n_chunks = (cols + 8 * NG - 1) / (8 * NG);
    const size_t smem = a.dot_mode == DOT_NONE ? 0 : size_t(kDmmaAnyWarps) * 2 * a.W * sizeof(double);
    const int64_t need = (a.n_block_rows * n_chunks + kDmmaAnyWarps - 1) / kDmmaAnyWarps;
    const int per_sm = occupancy(reinterpret_cast<const void*>(kernel), threads, smem);
    int64_t grid = int64_t(ctx->sm_count) * per_sm;
    if (grid > int64_t(ctx->sm_count) * 8) grid = int64_t(ctx->sm_count) * 8;
    if (need < grid) grid = need;
    if (grid < 1) grid = 1;
    kernel<<<unsigned(grid), threads, smem, ctx->stream>>>(a, n_chunks);
    RSATB_LAUNCH_CHECK(ctx);
    return RSATB_SUCCESS;
}

template <typename VT, int B, bool CM, bool CV, int... NGS>
int launch_dmma_any_b(rsatb_context* ctx, int groups, StepArgs& a) {
    // 2-value loads of the operand start on a boundary of their size.
    const bool pair_ok =
        a.W % 2 == 0 && (reinterpret_cast<uintptr_t>(a.in) & (2 * sizeof(VT) - 1)) == 0;
    int st = kNotApplicable;
    const auto with = [&](auto ng) {
        constexpr int NG = decltype(ng)::value;
        if (NG != groups) return false;
        if constexpr (CM) {
            if constexpr (B != 5)
                if (a.block_size <= 4) {
                    st = launch_dmma_any_k<VT, B, NG, 1, CM, CV, false>(ctx, a);
                    return true;
                }
            st = launch_dmma_any_k<VT, B, NG, 2, CM, CV, false>(ctx, a);
        } else {
            if constexpr (NG % 2 == 0)
                if (pair_ok) {
                    st = launch_dmma_any_k<VT, B, NG, 1, CM, CV, true>(ctx, a);
                    return true;
                }
            st = launch_dmma_any_k<VT, B, NG, 1, CM, CV, false>(ctx, a);
        }
        return true;
    };
    (with(std::integral_constant<int, NGS>()) || ...);
    return st;
}

// Column groups of 8 per warp: a panel of up to 64 columns is one warp's (b = 5
// and 8, the block sizes in use), wider ones split into chunks of 32; other
// block sizes take chunks of 8, 16 or 32.  Dots' shared memory: 4 warps x 2 x W
// doubles, 16 KB at W = 256.
template <typename VT, bool CM, bool CV>
int launch_dmma_any(rsatb_context* ctx, StepArgs& a) {
    if (a.block_size < 2 || a.block_size > 8 || a.W > 256) return kNotApplicable;
    const int groups = ((CM ? a.W / 2 : a.W) + 7) / 8;
    const int wide = groups <= 4 ? groups : groups <= 6 ? 6 : groups <= 8 ? 8 : 4;
    if (a.block_size == 5)
        return launch_dmma_any_b<VT, 5, CM, CV, 1, 2, 3, 4, 6, 8>(ctx, wide, a);
    if constexpr (!CM)
        if (a.block_size == 8)
            return launch_dmma_any_b<VT, 8, CM, CV, 1, 2, 3, 4, 6, 8>(ctx, wide, a);
    return launch_dmma_any_b<VT, 0, CM, CV, 1, 2, 4>(ctx, groups <= 2 ? groups : 4, a);
}

}  // namespace step_detail
}  // namespace rsatb_b200
