// Blocked FP64 Cholesky of one small symmetric positive definite system per
// warp on the FP64 tensor instruction (mma.sync m8n8k4).
//
// A system of up to 8 NB unknowns is held as 8x8 blocks of its lower triangle,
// each block in the accumulator layout of the instruction: lane 4 r + q holds
// entries (r, 2q) and (r, 2q+1). An m8n8k4 product sums over four of the eight
// columns, and the order of a sum over k is free as long as both operands use
// the same: taking the even columns first and the odd ones second, the .x and
// .y of an accumulator block are the two A operands and the two B operands of
// a product X Y^T. So the factorisation
//     L_ik = A_ik L_kk^-T,   A_ij -= L_ik L_jk^T
// needs no data movement between its steps: every product it makes is of the
// form X Y^T, with L_kk^-1 (M, below) formed explicitly per 8x8 diagonal block.
// Right-hand sides are carried as rows of one more block row X (rows 0..2 in
// use), which leaves X_k = (L^-1 rhs)^T and the forms rhs_i^T A^-1 rhs_j as the
// entries of sum_k X_k X_k^T.
#pragma once
#include <cuda_runtime.h>

namespace hb
{
struct Blk
{
    double x, y; // entries (r, 2q), (r, 2q+1) of an 8x8 block, lane = 4 r + q
};

__device__ __forceinline__ void mma884(Blk &c, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c.x), "+d"(c.y)
        : "d"(a), "d"(b));
}
// the product alone
__device__ __forceinline__ Blk mma884_zero(double a, double b)
{
    Blk c;
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%4};"
        : "=d"(c.x), "=d"(c.y)
        : "d"(a), "d"(b), "d"(0.0));
    return c;
}
// X Y^T
__device__ __forceinline__ Blk blk_prod_t(const Blk &x, const Blk &y)
{
    Blk c = mma884_zero(x.x, y.x);
    mma884(c, x.y, y.y);
    return c;
}
// C += X Y^T
__device__ __forceinline__ void blk_mul_t(Blk &c, const Blk &x, const Blk &y)
{
    mma884(c, x.x, y.x);
    mma884(c, x.y, y.y);
}
__device__ __forceinline__ double flip_sign(double v)
{
    return __hiloint2double(__double2hiint(v) ^ (int)0x80000000, __double2loint(v));
}
__device__ __forceinline__ Blk blk_neg(const Blk &b) { return Blk{flip_sign(b.x), flip_sign(b.y)}; }

// 1 / d for a positive normal pivot: the hardware's first approximation x0
// (relative error e, |e| < 2^-19) and one step of the third-order iteration
// x0 (1 + e + e^2), which leaves e^3 below the rounding of the last fma.
__device__ __forceinline__ double pivot_inverse(double d)
{
    double x0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x0) : "d"(d));
    const double e = fma(-d, x0, 1.0);
    return fma(x0, fma(e, e, e), x0);
}

// whether a pivot is not positive (or NaN), read off its exponent word; with
// EPS, whether it is below the machine epsilon 2^-52
template <bool EPS>
__device__ __forceinline__ bool pivot_fails(double d)
{
    const unsigned lo = EPS ? 0x3CB00000u : 1u;
    return (unsigned)__double2hiint(d) - lo >= 0x7FF00000u - lo;
}

// doubles of shared memory that mma_diag needs per system: two pairs of rows
constexpr int kMmaRowDoubles = 32;

// Factors the 8x8 diagonal blocks D[s] = L L^T of S systems (each warp-wide)
// and replaces them with M = L^-1 (zero above the diagonal). The elimination
// runs in place, two pivots a step: rows j and j + 1 are final at their step,
// and each later row r subtracts its multiples of both, whose slots hold M left
// of the pivots and D right of them; slots j and j + 1 of row r then start
// M(r, j) and M(r, j + 1), minus the multipliers. The two rows travel through
// shared memory (row: kMmaRowDoubles doubles per system, 16-byte aligned), which
// with the two reciprocals is the latency of a step (one pivot a step: twice the
// exchanges for a quarter fewer FP64 operations; the 8.3M systems of 32 then
// took 20.5 against 18.8 ms), and D(r, j) is read as D(j, r). The row scales
// d^-1/2 wait for the end, where the eight pivots take one rsqrt together.
// fail[s] is set (on every lane) by a pivot that is not positive, or, with
// EPS_PIVOT, below the machine epsilon. No step branches, so the chains of the S
// systems overlap.
template <int S, bool EPS_PIVOT>
__device__ __forceinline__ void mma_pivots(int j, Blk (&D)[S], double *row, int lane, bool (&fail)[S])
{
    const int r = lane >> 2, q = lane & 3;
    double *buf = row + (j & 2) * 8;
#pragma unroll
    for (int s = 0; s < S; ++s)
        if (r == j || r == j + 1)
            reinterpret_cast<double2 *>(buf + s * kMmaRowDoubles + 8 * (r & 1))[q] = make_double2(D[s].x, D[s].y);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < S; ++s)
    {
        const double *b0 = buf + s * kMmaRowDoubles, *b1 = b0 + 8;
        const double2 ab = reinterpret_cast<const double2 *>(b0)[j / 2]; // D(j, j), D(j, j + 1)
        const double ia = pivot_inverse(ab.x);
        const double t = ab.y * ia;
        const double d = fma(-t, ab.y, b1[j + 1]); // the second pivot
        fail[s] |= pivot_fails<EPS_PIVOT>(ab.x) || pivot_fails<EPS_PIVOT>(d);
        if (j == 6)
        {
            // no later rows: row 7 alone
            const double2 u0 = reinterpret_cast<const double2 *>(b0)[q];
            const double n0 = r == 7 ? t : 0.0;
            D[s].x = r == 7 && q == 3 ? -t : fma(-n0, u0.x, D[s].x);
            D[s].y = fma(-n0, u0.y, D[s].y);
            continue;
        }
        const double id = pivot_inverse(d);
        const double2 u0 = reinterpret_cast<const double2 *>(b0)[q], u1 = reinterpret_cast<const double2 *>(b1)[q];
        const double m0 = b0[r] * ia;
        const double m1 = r > j + 1 ? fma(-m0, ab.y, b1[r]) * id : 0.0;
        const double n0 = r > j + 1 ? fma(-m1, t, m0) : (r == j + 1 ? t : 0.0);
        const bool own = q == j / 2;
        D[s].x = own && r > j ? -n0 : fma(-m1, u1.x, fma(-n0, u0.x, D[s].x));
        D[s].y = own && r > j + 1 ? -m1 : fma(-m1, u1.y, fma(-n0, u0.y, D[s].y));
    }
}

// ROLL: the four steps as one copy of the code. For the sharing kernel, which is
// longer than the instruction cache likes (9.5M systems of up to 64: 62.3 -> 58.7 ms,
// 19.7M of up to 32: 21.9 -> 20.4 ms); the simulation's weights, a short loop, lose
// by it (8.3M systems: 23 -> 27 ms).
template <int S, bool EPS_PIVOT = false, bool ROLL = false>
__device__ __forceinline__ void mma_diag(Blk (&D)[S], double *row, int lane, bool (&fail)[S])
{
    const int r = lane >> 2, q = lane & 3;
    if constexpr (ROLL)
    {
#pragma unroll 1
        for (int j = 0; j < 8; j += 2) mma_pivots<S, EPS_PIVOT>(j, D, row, lane, fail);
    }
    else
    {
#pragma unroll
        for (int j = 0; j < 8; j += 2) mma_pivots<S, EPS_PIVOT>(j, D, row, lane, fail);
    }
#pragma unroll
    for (int s = 0; s < S; ++s)
    {
        const double own = (r & 1) ? D[s].y : D[s].x; // the pivot, in lane (r, r / 2)
        const double rs = rsqrt(__shfl_sync(0xffffffffu, own, (r << 2) + (r >> 1)));
        D[s].x = 2 * q < r ? D[s].x * rs : (2 * q == r ? rs : 0.0);
        D[s].y = 2 * q + 1 < r ? D[s].y * rs : (2 * q + 1 == r ? rs : 0.0);
    }
}

// index of block (i, k), i >= k, of the lower triangle
__host__ __device__ constexpr int blk_at(int i, int k) { return i * (i + 1) / 2 + k; }

// The factorisation with the forward substitution of the rows of X. A's
// diagonal blocks end as L_kk^-1, the others as L_ik, and X_k as
// (L^-1 rhs)^T. Block rows from nb on (warp-uniform) are skipped.
template <int NB, int S, bool EPS_PIVOT = false>
__device__ __forceinline__ void mma_factor(Blk (&A)[S][NB * (NB + 1) / 2], Blk (&X)[S][NB], int nb, double *row,
                                           int lane, bool (&fail)[S])
{
#pragma unroll
    for (int k = 0; k < NB; ++k)
    {
        if (k >= nb) break;
        Blk D[S];
#pragma unroll
        for (int s = 0; s < S; ++s) D[s] = A[s][blk_at(k, k)];
        mma_diag<S, EPS_PIVOT>(D, row, lane, fail);
#pragma unroll
        for (int s = 0; s < S; ++s)
        {
            A[s][blk_at(k, k)] = D[s];
            X[s][k] = blk_prod_t(X[s][k], D[s]);
        }
#pragma unroll
        for (int i = k + 1; i < NB; ++i)
        {
            if (i >= nb) break;
#pragma unroll
            for (int s = 0; s < S; ++s)
            {
                A[s][blk_at(i, k)] = blk_prod_t(A[s][blk_at(i, k)], D[s]);
            }
        }
#pragma unroll
        for (int j = k + 1; j < NB; ++j)
        {
            if (j >= nb) break;
#pragma unroll
            for (int s = 0; s < S; ++s)
            {
                const Blk n = blk_neg(A[s][blk_at(j, k)]);
                blk_mul_t(X[s][j], X[s][k], n);
#pragma unroll
                for (int i = j; i < NB; ++i)
                {
                    if (i >= nb) break;
                    blk_mul_t(A[s][blk_at(i, j)], A[s][blk_at(i, k)], n);
                }
            }
        }
    }
}

// The factorisation alone.
template <int NB, int S>
__device__ __forceinline__ void mma_factor(Blk (&A)[S][NB * (NB + 1) / 2], int nb, double *row, int lane,
                                           bool (&fail)[S])
{
#pragma unroll
    for (int k = 0; k < NB; ++k)
    {
        if (k >= nb) break;
        Blk D[S];
#pragma unroll
        for (int s = 0; s < S; ++s) D[s] = A[s][blk_at(k, k)];
        mma_diag<S, false, true>(D, row, lane, fail);
#pragma unroll
        for (int s = 0; s < S; ++s) A[s][blk_at(k, k)] = D[s];
#pragma unroll
        for (int i = k + 1; i < NB; ++i)
        {
            if (i >= nb) break;
#pragma unroll
            for (int s = 0; s < S; ++s)
            {
                A[s][blk_at(i, k)] = blk_prod_t(A[s][blk_at(i, k)], D[s]);
            }
        }
#pragma unroll
        for (int j = k + 1; j < NB; ++j)
        {
            if (j >= nb) break;
#pragma unroll
            for (int s = 0; s < S; ++s)
            {
                const Blk n = blk_neg(A[s][blk_at(j, k)]);
#pragma unroll
                for (int i = j; i < NB; ++i)
                {
                    if (i >= nb) break;
                    blk_mul_t(A[s][blk_at(i, j)], A[s][blk_at(i, k)], n);
                }
            }
        }
    }
}

// Loads the lower-triangle blocks of a covariance system: entry (i, c) is
// pair_c[|lin[i] - lin[c]|] (a displacement and its negative have the same
// covariance bit for bit, so one half of the table, and of the L1 footprint,
// is enough; pair_c: the pair table at offset zero; lin: the
// unknowns' table offsets, in shared memory, any value beyond n), the identity
// beyond the n live unknowns. UPPER leaves out the diagonal blocks' entries below
// the diagonal, which mma_diag does not read (D(r, j) is read as D(j, r)): with the
// analytic table of cokriging, whose gathers miss L1, 1.82M systems take 7.1 ms in
// place of 7.8; elsewhere it gains nothing and costs registers.
template <int NB, bool UPPER = false>
__device__ __forceinline__ void mma_load(Blk (&A)[NB * (NB + 1) / 2], const double *__restrict__ pair_c,
                                         const int *lin, int n, int nb, int lane)
{
    const int r = lane >> 2, q = lane & 3;
    int2 lc[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) lc[k] = reinterpret_cast<const int2 *>(lin + 8 * k)[q];
#pragma unroll
    for (int i = 0; i < NB; ++i)
    {
        if (i >= nb) break;
        const int row = 8 * i + r;
        const int rl = lin[row];
        if (8 * i + 8 <= n) // warp-uniform: every row of the block row is live
        {
#pragma unroll
            for (int k = 0; k <= i; ++k)
            {
                Blk &b = A[blk_at(i, k)];
                const bool all = !UPPER || k < i;
                b = Blk{0.0, 0.0};
                if (all || 2 * q >= r) b.x = __ldg(pair_c + abs(rl - lc[k].x));
                if (all || 2 * q + 1 >= r) b.y = __ldg(pair_c + abs(rl - lc[k].y));
            }
            continue;
        }
        const bool live = row < n;
#pragma unroll
        for (int k = 0; k < i; ++k)
        {
            Blk &b = A[blk_at(i, k)];
            b.x = live ? __ldg(pair_c + abs(rl - lc[k].x)) : 0.0;
            b.y = live ? __ldg(pair_c + abs(rl - lc[k].y)) : 0.0;
        }
        // the diagonal block whole (its two triangles are eliminated alike)
        const int c = 8 * i + 2 * q;
        Blk &b = A[blk_at(i, i)];
        b.x = (UPPER ? row <= c : live) && c < n ? __ldg(pair_c + abs(rl - lc[i].x)) : (row == c ? 1.0 : 0.0);
        b.y = (UPPER ? row <= c + 1 : live) && c + 1 < n ? __ldg(pair_c + abs(rl - lc[i].y)) : (row == c + 1 ? 1.0 : 0.0);
    }
}
} // namespace hb
