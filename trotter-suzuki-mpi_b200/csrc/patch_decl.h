// Entry points of the separately compiled register-patch steps
// (patch_f{64,32}_{real,imag}.cu) and their geometry.
#pragma once
#include <cuda_runtime.h>

#include "step_kernel.cuh"

namespace tsb {

// Blocks of 256 threads resident per SM that the registers are allocated for.
constexpr int patch_blocks(int n, bool fp32) { return fp32 ? (n == 2 ? 4 : 3) : (n == 2 ? 3 : 2); }

// The same for several steps per launch, whose tables of 2 x 2 patches stay in
// registers.
constexpr int patch_steps_blocks(int n, bool fp32) { return fp32 && n == 2 ? 4 : 2; }

// Cells per side that a region of 16 x 16 patches of n x n cells writes with
// a halo of h cells per sweep direction (whole patches).
constexpr int patch_out(int n, int h) { return 16 * n - 2 * ((h + n - 1) / n * n); }

// Regions up to which patches of 2 x 2 cells, and past those of 4 x 4 (0: never),
// take a tile's step on a GPU of `sms` SMs; pair: one species of two.  The limits
// were measured on 148 SMs (patch_cells in ts_b200.cu): places and turns of the
// regions go by the SMs.
struct PatchLimits {
    int side2, side4;
};
constexpr PatchLimits patch_limits(bool fp32, bool imag, bool rot, bool cyl, bool pair, bool phase,
                                   int sms) {
    const PatchLimits m = pair   ? PatchLimits{fp32 ? 520 : 750, 0}
                          : rot  ? PatchLimits{320, fp32 ? 2000 : 870}
                          : cyl  ? PatchLimits{260, fp32 ? 1100 : 300}
                          : fp32 ? PatchLimits{1100, imag ? 900 : 430}
                                 : PatchLimits{imag || !phase ? 1600 : 2100, 0};
    return PatchLimits{m.side2 * sms / 148, m.side4 * sms / 148};
}
static_assert(patch_limits(false, false, false, false, false, true, 148).side2 == 2100 &&
                  patch_limits(false, false, false, false, false, true, 74).side2 == 1050 &&
                  patch_limits(true, false, true, false, false, true, 74).side4 == 1000,
              "half the SMs, half the regions");

// n: cells of a thread's patch per side (2 or 4); phase as for the row walks
// (| 16: potential rows); pdl: programmatic dependent launch.
cudaError_t launch_patch_f64_real(int n, bool rot, int phase, const StepArgs<double> &a,
                                  int blocks, cudaStream_t st, bool pdl);
cudaError_t launch_patch_f64_imag(int n, bool rot, int phase, const StepArgs<double> &a,
                                  int blocks, cudaStream_t st, bool pdl);
cudaError_t launch_patch_f32_real(int n, bool rot, int phase, const StepArgs<float> &a,
                                  int blocks, cudaStream_t st, bool pdl);
cudaError_t launch_patch_f32_imag(int n, bool rot, int phase, const StepArgs<float> &a,
                                  int blocks, cudaStream_t st, bool pdl);

// m steps per launch of a closed tile in real time: phase 0, 1 or 2; patches
// of 2 x 2 cells with m = 2 or 3, of 4 x 4 with m = 2.
cudaError_t launch_patch_steps(int n, int m, int phase, const StepArgs<double> &a, int blocks,
                               cudaStream_t st, bool pdl);
cudaError_t launch_patch_steps(int n, int m, int phase, const StepArgs<float> &a, int blocks,
                               cudaStream_t st, bool pdl);

}  // namespace tsb
