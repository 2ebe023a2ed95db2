// The adjoint pass on register patches.
#include "adjoint_patch_decl.h"

#include "adjoint_patch.cuh"

namespace tsb {

namespace {
template <int MODE, int PHASE>
cudaError_t launch(const AdjArgs &a, int blocks, cudaStream_t st, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, adj_patch_kernel<AdjVariant<MODE, PHASE>, kAdjPatch>, a);
}

template <int MODE>
cudaError_t launch_mode(int phase, const AdjArgs &a, int blocks, cudaStream_t st, bool pdl) {
    if (phase == 2) return launch<MODE, 2>(a, blocks, st, pdl);
    if (phase == 1) return launch<MODE, 1>(a, blocks, st, pdl);
    return launch<MODE, 0>(a, blocks, st, pdl);
}
}  // namespace

cudaError_t launch_adj_patch(int mode, int phase, const AdjArgs &a, int blocks, cudaStream_t st,
                             bool pdl) {
    if (mode == 0) return launch<0, 0>(a, blocks, st, pdl);
    if (mode == 1) return launch_mode<1>(phase, a, blocks, st, pdl);
    return launch_mode<2>(phase, a, blocks, st, pdl);
}

}  // namespace tsb
