// gmle_corners.h - whether a ROI lies inside the calibration maps.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define GMLE_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define GMLE_HOST_DEVICE inline
#endif

namespace gmle {

// A box x box ROI at the 1-based corner (x, y) in maps of ny rows and nx columns.
// Any corner may stand in a caller's device arrays, which the host cannot check:
// the box is taken from the map's side (ny, nx >= 0, box <= 64), since x + box - 1
// overflows for a corner near the largest int32.
GMLE_HOST_DEVICE bool corner_inside(int32_t x, int32_t y, int32_t box, int32_t ny, int32_t nx)
{
    return x >= 1 && y >= 1 && x <= nx - box + 1 && y <= ny - box + 1;
}

}  // namespace gmle
