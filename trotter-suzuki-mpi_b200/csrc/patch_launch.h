// Launch templates of the register-patch step (patch.cuh); one translation
// unit per precision and time mode (patch_f{64,32}_{real,imag}.cu).
#pragma once
#include "patch.cuh"

namespace tsb {

template <class S>
cudaError_t launch_patch_shape(const StepArgs<typename S::T> &a, int blocks, cudaStream_t st,
                               bool pdl) {
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
    return cudaLaunchKernelEx(&cfg, patch_kernel<S>, a);
}

template <typename T, bool IMAG, bool ROT, int PHASE>
cudaError_t launch_patch_variant(int n, const StepArgs<T> &a, int blocks, cudaStream_t st,
                                 bool pdl) {
    using V = Variant<T, 2, IMAG, ROT, PHASE>;
    if (n == 2) return launch_patch_shape<PatchShape<V, 2>>(a, blocks, st, pdl);
    // only where patch_cells can choose them
    if constexpr (patch_limits(sizeof(T) == 4, IMAG, ROT, V::CYL, V::PB, V::PHASE, 148).side4 > 0)
        if (n == 4) return launch_patch_shape<PatchShape<V, 4>>(a, blocks, st, pdl);
    return cudaErrorInvalidValue;
}

template <typename T, bool IMAG>
cudaError_t launch_patch_t(int n, bool rot, int phase, const StepArgs<T> &a, int blocks,
                           cudaStream_t st, bool pdl) {
    if (rot) {
        if (phase == 0) return launch_patch_variant<T, IMAG, true, 0>(n, a, blocks, st, pdl);
        if (phase == 1) return launch_patch_variant<T, IMAG, true, 1>(n, a, blocks, st, pdl);
        if (phase == 2) return launch_patch_variant<T, IMAG, true, 2>(n, a, blocks, st, pdl);
        return cudaErrorInvalidValue;
    }
    if constexpr (!IMAG) {
        if (phase == 7) return launch_patch_variant<T, IMAG, false, 11>(n, a, blocks, st, pdl);
        if constexpr (sizeof(T) == 8) {
            if (phase == 16) return launch_patch_variant<T, IMAG, false, 16>(n, a, blocks, st, pdl);
            if (phase == 17) return launch_patch_variant<T, IMAG, false, 17>(n, a, blocks, st, pdl);
            if (phase == 18) return launch_patch_variant<T, IMAG, false, 18>(n, a, blocks, st, pdl);
        }
    }
    switch (phase) {
        case 0: return launch_patch_variant<T, IMAG, false, 0>(n, a, blocks, st, pdl);
        case 1: return launch_patch_variant<T, IMAG, false, 1>(n, a, blocks, st, pdl);
        case 2: return launch_patch_variant<T, IMAG, false, 2>(n, a, blocks, st, pdl);
        case 3: return launch_patch_variant<T, IMAG, false, 3>(n, a, blocks, st, pdl);
        case 4: return launch_patch_variant<T, IMAG, false, 4>(n, a, blocks, st, pdl);
        case 5: return launch_patch_variant<T, IMAG, false, 5>(n, a, blocks, st, pdl);
        case 6: return launch_patch_variant<T, IMAG, false, 6>(n, a, blocks, st, pdl);
    }
    return cudaErrorInvalidValue;
}

}  // namespace tsb
