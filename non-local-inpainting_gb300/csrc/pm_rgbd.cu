// PatchMatch kernels of the RGB-D distance.
#define NLI_PM_INSTANTIATE
#include "pm_kernels.cuh"

namespace nli {

template struct PmKernels<NLI_DIST_L2_RGBD, 4>;

NLI_CHECK_READER(check_word_pm_rgbd)

}  // namespace nli
