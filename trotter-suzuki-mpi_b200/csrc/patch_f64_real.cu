// Register-patch steps: double, real time.
#include "patch_launch.h"

namespace tsb {

cudaError_t launch_patch_f64_real(int n, bool rot, int phase, const StepArgs<double> &a, int blocks,
                                  cudaStream_t st, bool pdl) {
    return launch_patch_t<double, false>(n, rot, phase, a, blocks, st, pdl);
}

}  // namespace tsb
