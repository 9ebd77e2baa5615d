// The launches of the resident sweeps' kernels with one number of planes per
// thread in one form. Each is a translation unit of its own
// (kernels_sor_cluster_p*.cu, kernels_sor_grid_p*.cu): a program reaches one or two of them, and a
// kernel's first launch loads its whole unit. With all of a form in one unit the
// first solve of a process waited 20 ms for it.
#pragma once

#include "sor_resident.cuh"

namespace vb {
namespace resident {

template <int PZ, int MODE, int KIND, int GUARD, bool GRID>
void launch_variant(const Shape& p, const Args& a, cudaStream_t s) {
    const auto kernel = k_sor_resident<PZ, MODE, KIND, GUARD, GRID>;
    static OncePerDevice once;
    once([&] {
        VB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit - 2048));
        if (!GRID) VB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    });
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(p.ctas));
    cfg.blockDim = dim3(unsigned(p.threads));
    cfg.dynamicSmemBytes = size_t(p.smem);
    cfg.stream = s;
    cudaLaunchAttribute attr;
    if (GRID) {
        attr.id = cudaLaunchAttributeCooperative;
        attr.val.cooperative = 1;
    } else {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = unsigned(p.ctas);
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
    }
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    count_launch();
    VB_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
}

template <int PZ, int MODE, bool GRID>
void launch_mode(int kind, int guard, const Shape& p, const Args& a, cudaStream_t s) {
    if constexpr (MODE == kMixed)
        if (kind == kMasked) return launch_variant<PZ, MODE, kMasked, 2, GRID>(p, a, s);
    if (kind != kUniform) return launch_variant<PZ, MODE, kGeneral, 2, GRID>(p, a, s);
    if constexpr (MODE != kTolerance) {
        if (guard == 0) return launch_variant<PZ, MODE, kUniform, 0, GRID>(p, a, s);
        if constexpr (!GRID)
            if (guard == 1) return launch_variant<PZ, MODE, kUniform, 1, GRID>(p, a, s);
    }
    launch_variant<PZ, MODE, kUniform, 2, GRID>(p, a, s);
}

template <int PZ, bool GRID>
void launch_planes(Mode mode, int kind, int guard, const Shape& p, const Args& a, cudaStream_t s) {
    switch (mode) {
        case kFixed: launch_mode<PZ, kFixed, GRID>(kind, guard, p, a, s); break;
        case kTolerance: launch_mode<PZ, kTolerance, GRID>(kind, guard, p, a, s); break;
        default: launch_mode<PZ, kMixed, GRID>(kind, guard, p, a, s); break;
    }
}

}  // namespace resident
}  // namespace vb
