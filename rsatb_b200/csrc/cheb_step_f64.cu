// FP64 instantiations of the fused Chebyshev step and the column dots.
#include "cheb_step_impl.cuh"

namespace rsatb_b200 {

int launch_cheb_step_f64(rsatb_context* ctx, const rsatb_bsr_matrix* A, int vec_dtype,
                         StepArgs args) {
    return step_detail::launch_step_precision<double>(ctx, A, vec_dtype, args);
}

bool step_takes_ax(const rsatb_bsr_matrix* A) {
    return A->block_size == 1 && step_detail::env_kernel() == 0;
}

int launch_coldot_f64(rsatb_context* ctx, int vec_dtype, int64_t n_rows, StepArgs args) {
    return step_detail::launch_coldot_precision<double>(ctx, vec_dtype, n_rows, args);
}

}  // namespace rsatb_b200
