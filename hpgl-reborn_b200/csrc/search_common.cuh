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

// Whether the cells of template-path bin (bxi, byi, bzi), with C informed cells in the
// 27 bins around and `own` in itself, go to the template scan: its k-th informed cell
// is then expected after k vol / C of the template's offsets, whereas the lane-a-cell
// search stages and scans the C candidates and has fewer warps the more they are. The
// line, k vol / C = C / 4, lies where both take the same on uniform data: 500,000 cells,
// radius 10 (20), ms by search / scan at 5 % informed 0.92 / 1.00 (2.97 / 2.68) with 16
// neighbours and 2.31 / 2.36 (4.08 / 4.00) with 64, at 10 % 1.09 / 0.80 and 2.42 /
// 1.46, at 30 % 1.50 / 0.65 and 1.51 / 0.82. Beside a cluster of points, a bin with less than half
// the mean density of its 27, the scan is long whatever C is.
__device__ __forceinline__ bool scan_is_shorter(const Geom &g, int bxi, int byi, int bzi, int C, int own)
{
    const float wx = (float)(min(g.nx, (bxi + 2) * g.rx) - max(0, (bxi - 1) * g.rx));
    const float wy = (float)(min(g.ny, (byi + 2) * g.ry) - max(0, (byi - 1) * g.ry));
    const float wz = (float)(min(g.nz, (bzi + 2) * g.rz) - max(0, (bzi - 1) * g.rz));
    return 4.0f * (float)g.k * wx * wy * wz < (float)C * (float)C && 54LL * own >= C;
}

// transformed coordinates of an offset from the bin corner, in float
__device__ __forceinline__ float4 surr_coords(const SurrDev &sd, int x, int y, int z)
{
    const float fx = (float)x, fy = (float)y, fz = (float)z;
    return make_float4(fmaf(sd.T[2], fz, fmaf(sd.T[1], fy, sd.T[0] * fx)),
                       fmaf(sd.T[5], fz, fmaf(sd.T[4], fy, sd.T[3] * fx)),
                       fmaf(sd.T[8], fz, fmaf(sd.T[7], fy, sd.T[6] * fx)), 0.0f);
}

// The candidates of the 27 bins around bin (bxi, byi, bzi), z, y and x nested, as
// one list: the three bins along x lie one after another in bin_pts, so the list
// is nine runs. Lanes 0 to 15 of a warp write the runs' offsets in the list (past
// the ninth: past every place) and their starts in bin_pts; returns the length.
__device__ __forceinline__ int candidate_runs(const Geom &g, int bxi, int byi, int bzi, const int *bin_start,
                                              const int *bin_cnt, int lane, int *pre, int *start)
{
    int bs = 0, bc = 0;
    if (lane < 9)
    {
        const int kk = bzi - 1 + lane / 3, jj = byi - 1 + lane % 3;
        if (jj >= 0 && kk >= 0 && jj < g.by && kk < g.bz)
        {
            const int row = (kk * g.by + jj) * g.bx;
            const int i0 = max(bxi - 1, 0), i1 = min(bxi + 1, g.bx - 1);
            bs = bin_start[row + i0];
            bc = bin_start[row + i1] + bin_cnt[row + i1] - bs;
        }
    }
    int incl = bc;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1)
    {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane < 16)
    {
        pre[lane] = lane < 9 ? incl - bc : 0x7fffffff;
        start[lane] = bs;
    }
    return __shfl_sync(0xffffffffu, incl, 8);
}

// the last of the nine runs whose offset in the list is <= i
__device__ __forceinline__ int run_of(const int *pre, int i)
{
    int b = pre[8] <= i ? 8 : 0;
#pragma unroll
    for (int st = 4; st > 0; st >>= 1)
        if (pre[b + st] <= i) b += st;
    return b;
}
} // namespace hb
