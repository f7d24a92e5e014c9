// Launches and FP32 instantiations of the any-shape tensor-core step.
#include "cheb_dmma_any_launch.cuh"

namespace rsatb_b200 {
namespace step_detail {

template int launch_dmma_any<float, false, false>(rsatb_context*, StepArgs&);
template int launch_dmma_any<float, false, true>(rsatb_context*, StepArgs&);
template int launch_dmma_any<float, true, true>(rsatb_context*, StepArgs&);

}  // namespace step_detail
}  // namespace rsatb_b200
