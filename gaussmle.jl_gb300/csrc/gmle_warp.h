// gmle_warp.h - launch of the fit with one warp per ROI (gmle_fit_warp.cu),
// which takes the boxes that the specialised kernels do not.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "gmle_fit_kernel.cuh"

namespace gmle {

constexpr int kLargeMinBox = 17, kLargeMaxBox = 64;

inline bool large_box(int box) { return box >= kLargeMinBox && box <= kLargeMaxBox; }

// Shared memory, floats per ROI: 10 tables of `box` entries, and beyond 32
// pixels (which no longer fit a warp's registers) the ROI's pixels and variances.
__host__ __device__ constexpr int warp_floats(int box, bool scmos)
{
    return 10 * box + (box > 32 ? box * box * (scmos ? 2 : 1) : 0);
}

// ROIs (warps) per block: up to four, with three blocks' shared memory on an SM.
inline int warp_rois_per_block(int box, bool scmos)
{
    const int per = (int)sizeof(float) * warp_floats(box, scmos);
    return std::max(1, std::min(4, 72 * 1024 / per));
}

// Plain launch of ceil(a.n / rois_per_block) blocks over `a` (a.tpr == 32).
template <int MODEL, bool SCMOS>
cudaError_t launch_warp_family(int box, const KernelArgs &a, int rois_per_block, cudaStream_t s);
#define GMLE_EXTERN_WARP(M, S) \
    extern template cudaError_t launch_warp_family<M, S>(int, const KernelArgs &, int, cudaStream_t);
GMLE_EXTERN_WARP(0, false) GMLE_EXTERN_WARP(1, false) GMLE_EXTERN_WARP(2, false)
GMLE_EXTERN_WARP(3, false) GMLE_EXTERN_WARP(0, true) GMLE_EXTERN_WARP(1, true)
GMLE_EXTERN_WARP(2, true) GMLE_EXTERN_WARP(3, true)
#undef GMLE_EXTERN_WARP

inline cudaError_t launch_fit_warp(int model, int box, bool scmos, const KernelArgs &a,
                                   int rois_per_block, cudaStream_t s)
{
    switch (model * 2 + (int)scmos) {
        case 0: return launch_warp_family<0, false>(box, a, rois_per_block, s);
        case 1: return launch_warp_family<0, true>(box, a, rois_per_block, s);
        case 2: return launch_warp_family<1, false>(box, a, rois_per_block, s);
        case 3: return launch_warp_family<1, true>(box, a, rois_per_block, s);
        case 4: return launch_warp_family<2, false>(box, a, rois_per_block, s);
        case 5: return launch_warp_family<2, true>(box, a, rois_per_block, s);
        case 6: return launch_warp_family<3, false>(box, a, rois_per_block, s);
        case 7: return launch_warp_family<3, true>(box, a, rois_per_block, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gmle
