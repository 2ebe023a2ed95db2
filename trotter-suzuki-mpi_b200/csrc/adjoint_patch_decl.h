// Entry point of the separately compiled adjoint pass on register patches
// (adjoint_patch.cu).
#pragma once
#include <cuda_runtime.h>

#include "patch_decl.h"

namespace tsb {

struct AdjArgs;

constexpr int kAdjPatch = 2;        // patch side
constexpr int kAdjPatchBlocks = 2;  // blocks of 256 threads resident per SM

// mode and phase as AdjVariant; n_strips x n_segs regions of
// patch_out(kAdjPatch, 4) cells per side.
cudaError_t launch_adj_patch(int mode, int phase, const AdjArgs &a, int blocks, cudaStream_t st,
                             bool pdl);

}  // namespace tsb
