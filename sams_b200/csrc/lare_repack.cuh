// lare_repack.cuh -- dense box buffers to and from a solve's padded rows on
// the device, so that a host transfer is one contiguous copy.
#pragma once

#include "lare_device.cuh"

namespace sams {

// Dense box buffer <-> padded device rows (to_padded = 1: dense -> padded).
static __global__ void k_repack(const double *__restrict__ src, double *__restrict__ dst, Geom g, int to_padded)
{
    const long long n = (long long)(g.nx + 5) * (g.ny + 5) * (g.nz + 5);
    const int ez = g.nz + 5;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        const long long row = t / ez;
        const long long p = row * g.sy + (g.zoff - 2) + (t - row * ez);
        if (to_padded)
            dst[p] = src[t];
        else
            dst[t] = src[p];
    }
}

}  // namespace sams
