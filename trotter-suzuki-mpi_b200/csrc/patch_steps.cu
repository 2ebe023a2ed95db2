// Register-patch kernels that take several steps per launch (real time).
#include "patch_launch.h"

namespace tsb {

namespace {

template <class S>
cudaError_t launch_shape(const StepArgs<typename S::T> &a, int blocks, cudaStream_t st, bool pdl) {
    if (blocks == 0) return cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)S::THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, patch_steps_kernel<S>, a);
}

template <typename T, int PHASE>
cudaError_t launch_variant(int n, int m, const StepArgs<T> &a, int blocks, cudaStream_t st,
                           bool pdl) {
    using V = Variant<T, 2, false, false, PHASE>;
    if (n == 2 && m == 2) return launch_shape<PatchShape<V, 2, 2>>(a, blocks, st, pdl);
    if (n == 2 && m == 3) return launch_shape<PatchShape<V, 2, 3>>(a, blocks, st, pdl);
    if (n == 4 && m == 2) return launch_shape<PatchShape<V, 4, 2>>(a, blocks, st, pdl);
    return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_t(int n, int m, int phase, const StepArgs<T> &a, int blocks, cudaStream_t st,
                     bool pdl) {
    switch (phase) {
        case 0: return launch_variant<T, 0>(n, m, a, blocks, st, pdl);
        case 1: return launch_variant<T, 1>(n, m, a, blocks, st, pdl);
        case 2: return launch_variant<T, 2>(n, m, a, blocks, st, pdl);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_patch_steps(int n, int m, int phase, const StepArgs<double> &a, int blocks,
                               cudaStream_t st, bool pdl) {
    return launch_t<double>(n, m, phase, a, blocks, st, pdl);
}
cudaError_t launch_patch_steps(int n, int m, int phase, const StepArgs<float> &a, int blocks,
                               cudaStream_t st, bool pdl) {
    return launch_t<float>(n, m, phase, a, blocks, st, pdl);
}

}  // namespace tsb
