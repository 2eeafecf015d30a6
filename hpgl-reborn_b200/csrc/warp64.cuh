// FP64 solves of up to 32 symmetric positive definite systems of covariances
// with explicit solutions, one system per warp (the simulation, cokriging and
// leave-one-out kernels): the factorisation and forward substitution of mma64.cuh, the factor's
// blocks kept in shared memory, and the back substitution from there.
//
// Measured against it on the 8.3M systems of the 256x256x128 simulation: four
// warps as a team whose diagonal blocks one warp factors, eight lanes a system,
// between named barriers, 29.5 ms (fewer instructions, but three warps waiting
// on the chain of pivots of the fourth).
#pragma once
#include "mma64.cuh"

namespace hb
{
constexpr int kWarpNB = 4, kWarpN = 32, kWarpBlocks = 10;

template <int Q, bool SCALE>
struct __align__(16) WarpSmem
{
    double LM[kWarpBlocks * 64]; // L_ik, and L_kk^-1 on the diagonal (16-byte chunks swizzled)
    double row[kMmaRowDoubles];  // mma_diag's
    double y[Q][kWarpN];         // right-hand sides, L^-1 rhs, then the solutions
    double sig[SCALE ? kWarpN : 2];
    int lin[kWarpN];             // pair-table offsets of the unknowns
};

// offset of the 16-byte chunk of (r, 2q) in a block
__device__ __forceinline__ int blk_chunk(int r, int q) { return 4 * r + (q ^ ((r >> 1) & 3)); }

// The factorisation of the warp's system A of nb block rows with the forward
// substitution of its Q right-hand sides, T.y in place (it must be visible).
// Returns whether a pivot failed. HALVES: for users that return FP64 numbers.
template <int Q, bool EPS_PIVOT, bool SCALE, bool HALVES = false>
__device__ __forceinline__ bool warp_eliminate(WarpSmem<Q, SCALE> &T, int lane, int nb, Blk (&A)[1][kWarpBlocks])
{
    constexpr int NB = kWarpNB;
    const int r = lane >> 2, q = lane & 3;
    Blk X[1][NB];
#pragma unroll
    for (int k = 0; k < NB; ++k)
    {
        X[0][k] = Blk{0.0, 0.0};
        if (r < Q)
        {
            const double2 v = reinterpret_cast<const double2 *>(&T.y[r][8 * k])[q];
            X[0][k] = Blk{v.x, v.y};
        }
    }
    bool fail[1] = {false};
    if constexpr (HALVES)
        half_factor<NB, true, true, false>(A[0], X[0], nb, T.row, lane, fail[0]);
    else
        mma_factor<NB, 1, EPS_PIVOT>(A, X, nb, T.row, lane, fail);
    double2 *LM = reinterpret_cast<double2 *>(T.LM);
    const int at = blk_chunk(r, q);
    __syncwarp(); // the previous system's reads of LM are done
#pragma unroll
    for (int i = 0; i < NB; ++i)
    {
        if (i >= nb) break;
#pragma unroll
        for (int k = 0; k <= i; ++k)
            LM[blk_at(i, k) * 32 + at] = make_double2(A[0][blk_at(i, k)].x, A[0][blk_at(i, k)].y);
        if (r < Q) reinterpret_cast<double2 *>(&T.y[r][8 * i])[q] = make_double2(X[0][i].x, X[0][i].y);
    }
    __syncwarp();
    return fail[0];
}

// The same for the system of n unknowns read from a pair table (nb = ceil(n / 8));
// T.lin (and T.sig) must be visible too. Its users return floats and categories,
// whose rounding hides the whole inverses' error (by halves, 8.3M systems 26.2 -> 30.4 ms).
template <int Q, bool EPS_PIVOT, bool SCALE, bool UPPER = false>
__device__ __forceinline__ bool warp_factor(WarpSmem<Q, SCALE> &T, int lane, int n, int nb,
                                            const double *__restrict__ pair_c)
{
    constexpr int NB = kWarpNB;
    const int r = lane >> 2, q = lane & 3;
    Blk A[1][kWarpBlocks];
    mma_load<NB, UPPER>(A[0], pair_c, T.lin, n, nb, lane);
    if constexpr (SCALE)
    {
        // A[i][c] = pair * (sig_i * sig_c) for live entries (padding rows: sig 1)
#pragma unroll
        for (int i = 0; i < NB; ++i)
        {
            if (i >= nb) break;
            const double si = T.sig[8 * i + r];
#pragma unroll
            for (int k = 0; k <= i; ++k)
            {
                const double2 sc = reinterpret_cast<const double2 *>(&T.sig[8 * k])[q];
                Blk &b = A[0][blk_at(i, k)];
                b.x = __dmul_rn(b.x, __dmul_rn(si, sc.x));
                b.y = __dmul_rn(b.y, __dmul_rn(si, sc.y));
            }
        }
    }
    return warp_eliminate<Q, EPS_PIVOT, SCALE>(T, lane, nb, A);
}

// The back substitution of the warp's own system, L^T x = y, T.y in place: lane
// 8 p + c sums the rows 2 p and 2 p + 1 of column c of each block.
template <int Q, bool SCALE>
__device__ __forceinline__ void warp_back(WarpSmem<Q, SCALE> &T, int lane, int nb)
{
    const int p = lane >> 3, c = lane & 7;
    const double *LM = T.LM;
    const int e0 = 2 * blk_chunk(2 * p, c >> 1) + (c & 1), e1 = 2 * blk_chunk(2 * p + 1, c >> 1) + (c & 1);
    auto sum = [](double v) {
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        return v + __shfl_xor_sync(0xffffffffu, v, 16);
    };
#pragma unroll
    for (int k = kWarpNB - 1; k >= 0; --k)
    {
        if (k >= nb) continue;
        double s[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) s[q] = 0.0;
#pragma unroll
        for (int i = k + 1; i < kWarpNB; ++i)
        {
            if (i >= nb) break;
            const double l0 = LM[blk_at(i, k) * 64 + e0], l1 = LM[blk_at(i, k) * 64 + e1];
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                const double2 v = reinterpret_cast<const double2 *>(&T.y[q][8 * i])[p];
                s[q] = fma(l1, v.y, fma(l0, v.x, s[q]));
            }
        }
        double v[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) v[q] = T.y[q][8 * k + c];
        if (k + 1 < kWarpNB && k + 1 < nb)
        {
#pragma unroll
            for (int q = 0; q < Q; ++q) v[q] -= sum(s[q]);
            __syncwarp();
            if (p == 0)
            {
#pragma unroll
                for (int q = 0; q < Q; ++q) T.y[q][8 * k + c] = v[q];
            }
            __syncwarp();
        }
        const double m0 = LM[blk_at(k, k) * 64 + e0], m1 = LM[blk_at(k, k) * 64 + e1];
        double x[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            const double2 r = reinterpret_cast<const double2 *>(&T.y[q][8 * k])[p];
            x[q] = sum(fma(m1, r.y, m0 * r.x));
        }
        __syncwarp();
        if (p == 0)
        {
#pragma unroll
            for (int q = 0; q < Q; ++q) T.y[q][8 * k + c] = x[q];
        }
        __syncwarp();
    }
}
} // namespace hb
