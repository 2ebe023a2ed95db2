// Register-patch steps: float, imaginary time.
#include "patch_launch.h"

namespace tsb {

cudaError_t launch_patch_f32_imag(int n, bool rot, int phase, const StepArgs<float> &a, int blocks,
                                  cudaStream_t st, bool pdl) {
    return launch_patch_t<float, true>(n, rot, phase, a, blocks, st, pdl);
}

}  // namespace tsb
