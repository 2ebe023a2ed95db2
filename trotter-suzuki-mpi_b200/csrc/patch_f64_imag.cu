// Register-patch steps: double, imaginary time.
#include "patch_launch.h"

namespace tsb {

cudaError_t launch_patch_f64_imag(int n, bool rot, int phase, const StepArgs<double> &a, int blocks,
                                  cudaStream_t st, bool pdl) {
    return launch_patch_t<double, true>(n, rot, phase, a, blocks, st, pdl);
}

}  // namespace tsb
