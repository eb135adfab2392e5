// gmle_warp.h - launch of the fit with one warp per ROI (gmle_fit_warp.cu): the
// boxes that the specialised kernels do not take, and small batches of the others.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "gmle_fit_kernel.cuh"

namespace gmle {

constexpr int kLargeMinBox = 17, kLargeMaxBox = 64;

inline bool large_box(int box) { return box >= kLargeMinBox && box <= kLargeMaxBox; }

// Rows per lane, RMAX = ceil(box / 4), of the kernel that takes a box.
__host__ __device__ constexpr int rows_per_lane(int box)
{
    return box <= 8 ? 2 : box <= 32 ? (box + 3) / 4 : box <= 48 ? 12 : 16;
}

// Shared memory, floats per ROI: 10 tables of 4 RMAX entries (a compile-time
// stride; the entries past the box stay 0), then up to 16 pixels three arrays of
// the ROI's pixels, for the start point's sums in the reference's order, and
// beyond 32, which no longer fit a warp's registers, pixels and variances.
__host__ __device__ constexpr int warp_scratch(int box) { return (box * box + 3) & ~3; }
__host__ __device__ constexpr int warp_floats(int box, bool scmos)
{
    return 40 * rows_per_lane(box) +
           (box <= 16 ? 3 * warp_scratch(box) : box > 32 ? warp_scratch(box) * (scmos ? 2 : 1) : 0);
}

// ROIs (warps) per block, up to four (their FP64 inversions share instructions):
// boxes up to 16 spread over the SMs, two blocks per SM or more (2000 XYNBS 9x9
// ROIs in blocks of six, two of which fit an SM's registers: 57 us, a second wave
// of 30 blocks; in blocks of four: 35 us); larger boxes with three blocks' shared
// memory on an SM.
constexpr int kWarpMaxRois = 4;
inline int warp_rois_per_block(int num_sms, int box, bool scmos, int64_t n)
{
    if (box <= 16)
        return (int)std::max<int64_t>(1, std::min<int64_t>(kWarpMaxRois, n / (2 * num_sms)));
    const int per = (int)sizeof(float) * warp_floats(box, scmos);
    return std::max(1, std::min(kWarpMaxRois, 72 * 1024 / per));
}

// Plain launch (t.header == nullptr) of ceil(a.n / rois_per_block) blocks over
// `a`, or a table launch of `grid` blocks (boxes up to 16), with a.tpr == 32.
template <int MODEL, bool SCMOS>
cudaError_t launch_warp_family(int box, const KernelArgs &a, const TileTable &t,
                               int rois_per_block, int64_t grid, cudaStream_t s);
// Resident blocks per SM of a table launch (a negated cudaError_t on error).
template <int MODEL, bool SCMOS> int warp_table_blocks(int box, int rois_per_block);
#define GMLE_EXTERN_WARP(M, S) \
    extern template cudaError_t launch_warp_family<M, S>(int, const KernelArgs &, const TileTable &, \
                                                         int, int64_t, cudaStream_t);             \
    extern template int warp_table_blocks<M, S>(int, int);
GMLE_EXTERN_WARP(0, false) GMLE_EXTERN_WARP(1, false) GMLE_EXTERN_WARP(2, false)
GMLE_EXTERN_WARP(3, false) GMLE_EXTERN_WARP(0, true) GMLE_EXTERN_WARP(1, true)
GMLE_EXTERN_WARP(2, true) GMLE_EXTERN_WARP(3, true)
#undef GMLE_EXTERN_WARP

inline cudaError_t launch_fit_warp(int model, int box, bool scmos, const KernelArgs &a,
                                   const TileTable &t, int rois_per_block, int64_t grid,
                                   cudaStream_t s)
{
#define GMLE_CASE(M)                                                                        \
    case M:                                                                                 \
        return scmos ? launch_warp_family<M, true>(box, a, t, rois_per_block, grid, s)      \
                     : launch_warp_family<M, false>(box, a, t, rois_per_block, grid, s);
    switch (model) {
        GMLE_CASE(0) GMLE_CASE(1) GMLE_CASE(2) GMLE_CASE(3)
        default: return cudaErrorInvalidValue;
    }
#undef GMLE_CASE
}

inline int warp_table_blocks_per_sm(int model, int box, bool scmos, int rois_per_block)
{
#define GMLE_CASE(M)                                                  \
    case M:                                                           \
        return scmos ? warp_table_blocks<M, true>(box, rois_per_block) \
                     : warp_table_blocks<M, false>(box, rois_per_block);
    switch (model) {
        GMLE_CASE(0) GMLE_CASE(1) GMLE_CASE(2) GMLE_CASE(3)
        default: return 0;
    }
#undef GMLE_CASE
}

}  // namespace gmle
