// Table of the fused substep kernel's instantiations for one scene source
// (FIXED: the scene from the kernel parameters, else from the device table),
// indexed by dimension, material and launch configuration (configurations
// that differ only in rounds or particle order share an instantiation).  Each source's
// table is instantiated in its own translation unit so they compile in
// parallel.
#pragma once

#include "mpm_dispatch.cuh"

namespace mpm {

// the run-sum kernel of launch shape K, when a configuration asks for it
template <int K, bool PAGED>
static constexpr bool has_runs() {
    for (int i = 0; i < kNumFusedCfgs; ++i)
        if (kFusedCfgs[i].kernel == K && sums_runs(i, PAGED)) return true;
    return false;
}

template <int D, int MAT, int K, bool FIXED, bool PAGED>
static FusedFn fused_kernel(bool runs) {
    constexpr FusedKernel k = kFusedKernels[K];
    if constexpr (has_runs<K, PAGED>())
        if (runs) return &k_g2p2g_runs<D, MAT, k.chunk, k.min_ctas, FIXED, PAGED>;
    if constexpr (k.scatter == SCATTER_DIRECT) return &k_g2p2g<D, MAT, k.chunk, k.min_ctas, FIXED, PAGED>;
    else return nullptr;  // declared run sums address a dense grid
}

template <int D, int MAT, bool FIXED, bool PAGED>
static FusedFn fused_for(int ci) {
    static_assert(kNumFusedKernels == 12, "update the dispatch table");
    const bool r = sums_runs(ci, PAGED);
    switch (kFusedCfgs[ci].kernel) {
        case 0: return fused_kernel<D, MAT, 0, FIXED, PAGED>(r);
        case 1: return fused_kernel<D, MAT, 1, FIXED, PAGED>(r);
        case 2: return fused_kernel<D, MAT, 2, FIXED, PAGED>(r);
        case 3: return fused_kernel<D, MAT, 3, FIXED, PAGED>(r);
        case 4: return fused_kernel<D, MAT, 4, FIXED, PAGED>(r);
        case 5: return fused_kernel<D, MAT, 5, FIXED, PAGED>(r);
        case 6: return fused_kernel<D, MAT, 6, FIXED, PAGED>(r);
        case 7: return fused_kernel<D, MAT, 7, FIXED, PAGED>(r);
        case 8: return fused_kernel<D, MAT, 8, FIXED, PAGED>(r);
        case 9: return fused_kernel<D, MAT, 9, FIXED, PAGED>(r);
        case 10: return fused_kernel<D, MAT, 10, FIXED, PAGED>(r);
        default: return fused_kernel<D, MAT, 11, FIXED, PAGED>(r);
    }
}

template <int D, bool FIXED, bool PAGED>
static FusedFn fused_for_mat(int mat, int ci) {
    if (mat == JELLO) return fused_for<D, JELLO, FIXED, PAGED>(ci);
    if (mat == SNOW) return fused_for<D, SNOW, FIXED, PAGED>(ci);
    return fused_for<D, WATER, FIXED, PAGED>(ci);
}

template <bool FIXED, bool PAGED>
static FusedFn fused_table(int dim, int mat, int ci) {
    return dim == 3 ? fused_for_mat<3, FIXED, PAGED>(mat, ci) : fused_for_mat<2, FIXED, PAGED>(mat, ci);
}

}  // namespace mpm
