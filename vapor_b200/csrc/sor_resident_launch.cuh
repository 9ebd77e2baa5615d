// The launches of the resident sweeps' kernels with one number of planes per
// thread in one form. Each is a translation unit of its own
// (kernels_sor_cluster_p*.cu, kernels_sor_grid_p*.cu): a program reaches one or two of them, and a
// kernel's first launch loads its whole unit. With all of a form in one unit the
// first solve of a process waited 20 ms for it.
#pragma once

#include "sor_resident.cuh"

namespace vb {
namespace resident {

// Whether the device can hold the launch: some devices have no cluster of that
// many SMs free (a partition of the GPU, for one).
template <int PZ, int MODE, int KIND, int GUARD, bool GRID>
bool fits(const Shape& p, const cudaLaunchConfig_t& cfg) {
    static std::mutex mutex;
    static std::map<std::tuple<int, int, int, int>, bool> known;
    int device = 0;
    VB_CUDA(cudaGetDevice(&device));
    const std::tuple<int, int, int, int> key(device, p.ctas, p.threads, p.smem);
    std::lock_guard<std::mutex> lock(mutex);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    const auto kernel = k_sor_resident<PZ, MODE, KIND, GUARD, GRID>;
    int most = 0, sms = 0;
    cudaError_t e;
    if (GRID) {
        VB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&most, kernel, p.threads, size_t(p.smem));
        most = most * sms >= p.ctas;
    } else {
        e = cudaOccupancyMaxActiveClusters(&most, kernel, &cfg);
    }
    if (e != cudaSuccess) cudaGetLastError();  // a shape that the device does not know
    return known[key] = e == cudaSuccess && most > 0;
}

// Launches the kernel, or with `query` only says whether the device can hold it.
template <int PZ, int MODE, int KIND, int GUARD, bool GRID>
bool launch_variant(const Shape& p, const Args& a, bool query, cudaStream_t s) {
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
    if (query) return fits<PZ, MODE, KIND, GUARD, GRID>(p, cfg);
    count_launch();
    VB_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    return true;
}

template <int PZ, int MODE, bool GRID>
bool launch_mode(int kind, int guard, const Shape& p, const Args& a, bool query, cudaStream_t s) {
    if constexpr (MODE == kMixed)
        if (kind == kMasked) return launch_variant<PZ, MODE, kMasked, 2, GRID>(p, a, query, s);
    if (kind != kUniform) return launch_variant<PZ, MODE, kGeneral, 2, GRID>(p, a, query, s);
    if constexpr (MODE != kTolerance) {
        if (guard == 0) return launch_variant<PZ, MODE, kUniform, 0, GRID>(p, a, query, s);
        if constexpr (!GRID)
            if (guard == 1) return launch_variant<PZ, MODE, kUniform, 1, GRID>(p, a, query, s);
    }
    return launch_variant<PZ, MODE, kUniform, 2, GRID>(p, a, query, s);
}

template <int PZ, bool GRID>
bool launch_planes(Mode mode, int kind, int guard, const Shape& p, const Args& a, bool query, cudaStream_t s) {
    switch (mode) {
        case kFixed: return launch_mode<PZ, kFixed, GRID>(kind, guard, p, a, query, s);
        case kTolerance: return launch_mode<PZ, kTolerance, GRID>(kind, guard, p, a, query, s);
        default: return launch_mode<PZ, kMixed, GRID>(kind, guard, p, a, query, s);
    }
}

}  // namespace resident
}  // namespace vb
