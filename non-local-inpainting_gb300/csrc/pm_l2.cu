// PatchMatch kernels of the L2 norm.
#define NLI_PM_INSTANTIATE
#include "pm_kernels.cuh"

namespace nli {

template struct PmKernels<NLI_DIST_L2_NORM, 1>;
template struct PmKernels<NLI_DIST_L2_NORM, 2>;
template struct PmKernels<NLI_DIST_L2_NORM, 3>;
template struct PmKernels<NLI_DIST_L2_NORM, 4>;

NLI_CHECK_READER(check_word_pm_l2)

}  // namespace nli
