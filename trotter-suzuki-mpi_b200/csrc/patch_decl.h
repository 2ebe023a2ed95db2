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
