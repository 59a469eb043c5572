// snap.cuh -- the pixel of a point and its Morton code (setup and the spatial sort).
#pragma once
#include "internal.cuh"

namespace galpha {

// Pixel of an input point inside the margin (the snap SetupSites makes).
__device__ __forceinline__ void snap_pixel(double x, double y, double sx, double sy, double scale, int D, int *ix,
                                           int *iy)
{
    const double gx = floor((x - sx) / scale), gy = floor((y - sy) / scale);
    *ix = (int)fmin(fmax(gx, 0.0), (double)(D - 1));
    *iy = (int)fmin(fmax(gy, 0.0), (double)(D - 1));
}

__device__ __forceinline__ unsigned spread_bits14(unsigned v)
{
    v &= 0x3fffu;
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}

__device__ __forceinline__ unsigned pixel_key(double x, double y, const SnapGrid &g)
{
    int ix, iy;
    snap_pixel(x, y, g.sx, g.sy, g.scale, g.D, &ix, &iy);
    return spread_bits14((unsigned)ix) | (spread_bits14((unsigned)iy) << 1);
}

}  // namespace galpha
