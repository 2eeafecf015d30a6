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
// form X Y^T. How L_kk^-1 is applied is a choice: as one explicit 8x8 inverse M
// (mma_factor), or by halves (half_factor). Right-hand sides are carried as rows of
// one more block row X (rows 0..2 in use), which leaves X_k = (L^-1 rhs)^T and the
// forms rhs_i^T A^-1 rhs_j as the entries of sum_k X_k X_k^T.
//
// Rounding. With M the error is that of a substitution times the condition of L_kk.
// Root mean square errors against 128 bits of the sharing solves (estimate and
// variance, simple kriging but for the clustered wells), relative to right-looking
// substitutions in order of falling covariance:
//                                         with M       by halves
//     Gaussian, nugget 0.05, 32       2.2   1.6     1.3   1.3
//     Gaussian, nugget 0.05, 24       3.0   1.5     1.5   1.1
//     Gaussian, nugget 0.001, clustered, 64     1.6   1.7     1.0   1.1
//     spherical, no nugget, 24        1.9   1.3     1.3   1.2
//     exponential, no nugget, 32      1.3   1.3     1.2   1.3
// (The absolute ones are 10^-16 to 10^-15, clustered 10^-13.) By halves is slower
// (half_diag), so the sharing solves take it where it shows: SolveOut::by_halves.
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

// 1 / d for a pivot that pivot_fails passes (d and 1 / d are then normal numbers):
// Chebyshev's third-order iteration on 1 / x = d (J. F. Traub, Iterative Methods for
// the Solution of Equations, 1964) from the hardware's approximation,
//     e = 1 - d x0,   x = x0 + x0 (e + e^2),   1 / d - x = e^3 / d.
// x0 comes from d's upper 32 bits and has as many (PTX manual): |e| < 2^-19, which
// leaves e^3 < 2^-57, a sixteenth of the last place beside the last fma's half: x is
// 1 / d rounded or the number next to it. (__drcp_rn, which branches for the extreme
// exponents: the sharing solves of 8.3M systems of 32 10.9 -> 12.4 ms, 8.3M
// simulation weights 26.4 -> 31.0 ms.)
__device__ __forceinline__ double pivot_inverse(double d)
{
    double x0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x0) : "d"(d));
    const double e = fma(-d, x0, 1.0);
    return fma(x0, fma(e, e, e), x0);
}

// whether a pivot is not positive (or NaN), or so small or large that d or 1 / d is
// no normal number (below 2^-1022, from 2^1022 on), read off its exponent word; with
// EPS, whether it is below the machine epsilon 2^-52
template <bool EPS>
__device__ __forceinline__ bool pivot_fails(double d)
{
    const unsigned lo = EPS ? 0x3CB00000u : 0x00100000u;
    return (unsigned)__double2hiint(d) - lo >= 0x7FD00000u - lo;
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

// The place of the i-th of n unknowns in order of importance (i < n): dealt out to
// the nb = ceil(n / 8) blocks in turn, so that neither a block nor a half of one
// holds unknowns that are nearly dependent. Places beyond n stay.
__device__ __forceinline__ int mma_slot(int i, int n, int nb)
{
    const float inv = __frcp_rn((float)nb); // quotients of less than 64 by at most 8
    const int j = (int)(((float)i + 0.5f) * inv), per = (int)(((float)n + 0.5f) * inv), k = i - j * nb;
    return i < n ? k * per + min(k, n - per * nb) + j : i;
}

// ---- by halves: the even slots are eliminated first, then the odd ones,
//     L_kk = [E 0; F O]:  X_e = A_e E^-1T,  X_o = (A_o - X_e F^T) O^-1T,
// with E^-1 and O^-1 (4x4) explicit: three dependent products in place of two, and
// the error of a substitution. The elimination is mma_diag's with the pivots
// p0 and p1 = p0 + 2: (0, 2) and (4, 6), then, ODD, (1, 3) and (5, 7) (h = 0 and 1).
// The sharing solves of 8.3M systems of 32 take 11.6 ms in place of 10.9, of 9.5M of
// up to 64 62.7 in place of 55.8.
struct Halves
{
    Blk half; // E^-1 in the even rows' x, -F in the odd rows' x, O^-1 in the odd rows' y, zero elsewhere
    Blk inv;  // with INV, L_kk^-1
};

__device__ __forceinline__ Blk blk_solve_t(const Blk &a, const Blk &half)
{
    const Blk e = mma884_zero(a.x, half.x);
    Blk c{0.0, a.y};
    mma884(c, e.x, half.x);
    return Blk{e.x, mma884_zero(c.y, half.y).y};
}

// INV: the odd rows' even columns are wanted too (they are part of the inverse alone)
template <bool INV, bool ODD>
__device__ __forceinline__ void half_pivots(int h, Blk &D, double *row, int lane, bool &fail)
{
    const int r = lane >> 2, q = lane & 3, p0 = 4 * h + ODD, p1 = p0 + 2;
    double2 *b = reinterpret_cast<double2 *>(row) + 8 * h; // b[c] = (D(p0, c), D(p1, c))
    if (r == p0 || r == p1)
    {
        double *w = reinterpret_cast<double *>(b + 2 * q) + (r == p1);
        if (!ODD || INV) w[0] = D.x;
        w[2] = D.y;
    }
    __syncwarp();
    const double2 s = b[p1];
    const double a = b[p0].x, ab = s.x, bb = s.y;
    const double ia = pivot_inverse(a);
    const double t = ab * ia;
    const double d = fma(-t, ab, bb); // the second pivot
    fail |= pivot_fails<false>(a) || pivot_fails<false>(d);
    const double id = pivot_inverse(d);
    const double2 v = b[r], uy = b[2 * q + 1];
    double2 ux = make_double2(0.0, 0.0);
    if (!ODD || INV) ux = b[2 * q];
    const bool later = ODD ? (r & 1) && r > p1 : (r & 1) || r > p1;
    const double m0 = v.x * ia;
    const double m1 = later ? fma(-m0, ab, v.y) * id : 0.0;
    const double n0 = later ? fma(-m1, t, m0) : (r == p1 ? t : 0.0);
    const bool own0 = q == p0 >> 1 && (later || r == p1), own1 = q == p1 >> 1 && later;
    if (!ODD || INV)
    {
        const double x = fma(-m1, ux.y, fma(-n0, ux.x, D.x));
        D.x = ODD ? x : (own0 ? -n0 : (own1 ? -m1 : x));
    }
    const double y = fma(-m1, uy.y, fma(-n0, uy.x, D.y));
    D.y = ODD ? (own0 ? -n0 : (own1 ? -m1 : y)) : y;
}

template <bool INV, bool ROLL>
__device__ __forceinline__ Halves half_diag(Blk D, double *row, int lane, bool &fail)
{
    const int r = lane >> 2, q = lane & 3;
    if constexpr (ROLL)
    {
#pragma unroll 1
        for (int h = 0; h < 2; ++h) half_pivots<INV, false>(h, D, row, lane, fail);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) half_pivots<INV, true>(h, D, row, lane, fail);
    }
    else
    {
#pragma unroll
        for (int h = 0; h < 2; ++h) half_pivots<INV, false>(h, D, row, lane, fail);
#pragma unroll
        for (int h = 0; h < 2; ++h) half_pivots<INV, true>(h, D, row, lane, fail);
    }
    const bool odd = r & 1;
    const double own = odd ? D.y : D.x; // the pivot, in lane (r, r / 2)
    const double rs = rsqrt(__shfl_sync(0xffffffffu, own, (r << 2) + (r >> 1)));
    const double x = D.x * rs, y = D.y * rs; // an even row's y: F^T
    const double f = __shfl_sync(0xffffffffu, y, 8 * q + (r >> 1));
    Halves o;
    const double ex = 2 * q < r ? x : (2 * q == r ? rs : 0.0);
    o.half.x = odd ? flip_sign(f) : ex;
    o.half.y = !odd || 2 * q + 1 > r ? 0.0 : (2 * q + 1 == r ? rs : y);
    o.inv = Blk{odd ? x : ex, o.half.y};
    return o;
}

// The factorisation by halves, with the forward substitution of the rows of X (RHS).
// A's diagonal blocks end as the half forms or, with INV, as the inverses.
template <int NB, bool RHS, bool INV, bool ROLL>
__device__ __forceinline__ void half_factor(Blk (&A)[NB * (NB + 1) / 2], Blk (&X)[RHS ? NB : 1], int nb, double *row,
                                            int lane, bool &fail)
{
#pragma unroll
    for (int k = 0; k < NB; ++k)
    {
        if (k >= nb) break;
        const Halves D = half_diag<INV, ROLL>(A[blk_at(k, k)], row, lane, fail);
        A[blk_at(k, k)] = INV ? D.inv : D.half;
        if constexpr (RHS) X[k] = blk_solve_t(X[k], D.half);
#pragma unroll
        for (int i = k + 1; i < NB; ++i)
        {
            if (i >= nb) break;
            A[blk_at(i, k)] = blk_solve_t(A[blk_at(i, k)], D.half);
        }
#pragma unroll
        for (int j = k + 1; j < NB; ++j)
        {
            if (j >= nb) break;
            const Blk n = blk_neg(A[blk_at(j, k)]);
            if constexpr (RHS) blk_mul_t(X[j], X[k], n);
#pragma unroll
            for (int i = j; i < NB; ++i)
            {
                if (i >= nb) break;
                blk_mul_t(A[blk_at(i, j)], A[blk_at(i, k)], n);
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
// the diagonal, which mma_diag (not half_diag) does not read: with the
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
