// Pieces shared by the neighbour searches (search.cu, search_tile.cu).
#pragma once
#include "engine.cuh"
#include "kernels.h"

namespace hb
{
__device__ __forceinline__ unsigned lanemask_lt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// transformed coordinates of an offset from the bin corner, in float
__device__ __forceinline__ float4 surr_coords(const SurrDev &sd, int x, int y, int z)
{
    const float fx = (float)x, fy = (float)y, fz = (float)z;
    return make_float4(fmaf(sd.T[2], fz, fmaf(sd.T[1], fy, sd.T[0] * fx)),
                       fmaf(sd.T[5], fz, fmaf(sd.T[4], fy, sd.T[3] * fx)),
                       fmaf(sd.T[8], fz, fmaf(sd.T[7], fy, sd.T[6] * fx)), 0.0f);
}
} // namespace hb
