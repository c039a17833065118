// PatchMatch kernels of the combined L2 distance on 3 channels.
#define NLI_PM_INSTANTIATE
#include "pm_kernels.cuh"

namespace nli {

template struct PmKernels<NLI_DIST_L2_COMBINED, 3>;

NLI_CHECK_READER(check_word_pm_combined_rgb)

}  // namespace nli
