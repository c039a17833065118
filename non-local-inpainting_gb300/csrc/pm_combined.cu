// PatchMatch kernels of the combined L2 distance on 1, 2 and 4 channels.
#define NLI_PM_INSTANTIATE
#include "pm_kernels.cuh"

namespace nli {

template struct PmKernels<NLI_DIST_L2_COMBINED, 1>;
template struct PmKernels<NLI_DIST_L2_COMBINED, 2>;
template struct PmKernels<NLI_DIST_L2_COMBINED, 4>;

NLI_CHECK_READER(check_word_pm_combined)

}  // namespace nli
