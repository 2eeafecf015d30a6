// Simple collocated cokriging, Markov models I and II
// (simple_cokriging_markI.cpp:19-330).
//
// Every uninformed cell is kriged from the first max_nb informed primary cells
// of the analytic search template (the kriging path's template search over the
// informed-cell bitmap, run for every bin) and the collocated secondary value. The bordered system
//   [ A   c ] [w ]   [ b   ]
//   [ c^T s ] [wn] = [ b_n ]
// (A, b: primary covariances; c: the cross covariances of the target with the
// neighbours; s: the secondary variance; b_n: the cross covariance at 0) is
// solved through A: x = A^-1 b, y = A^-1 c, then wn = (b_n - c.x) / (s - c.y)
// and w = x - wn y, the same solution as the reference's Gaussian elimination
// (gauss_solver.cpp:8-70), which processes the border last. The result is
// combine()'s float accumulation (simple_cokriging_markI.cpp:83-106).
#include "engine.cuh"
#include "kernels.h"
#include "warp64.cuh"

#include <algorithm>
#include <cfloat>
#include <climits>

namespace hb
{
// flag[i] = 1 for the targets (uninformed primary cells)
__global__ void k_cok_prepare(long long n, const uint8_t *__restrict__ pmask, int *__restrict__ flag)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        flag[i] = pmask[i] ? 0 : 1;
}

__global__ void k_cok_targets(long long n, const int *__restrict__ flag, const int *__restrict__ pos,
                              int *__restrict__ targets)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        if (flag[i]) targets[pos[i]] = (int)i;
}

// informed cells copy the primary value (every output cell ends informed)
__global__ void k_cok_finalize(long long n, const float *__restrict__ pdata, const uint8_t *__restrict__ pmask,
                               float *__restrict__ out_data, uint8_t *__restrict__ out_mask,
                               signed char *__restrict__ status)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        if (pmask[i])
        {
            out_data[i] = pdata[i];
            out_mask[i] = 1;
            if (status) status[i] = -1;
        }
}

struct CokArgsDev
{
    Geom g;
    const int *targets;
    int n_targets;
    const int2 *nb_rec; // per cell and slot: {pair-table offset, value bits}
    const int *nb_n;    // per cell
    int k;
    const double *pair64;
    const double *cross_tab;
    const float *pdata;
    const float *sdata;
    const uint8_t *smask;
    CokParams p;
    float *out_data;
    uint8_t *out_mask;
    signed char *status;
};

// the cross table's entry of a neighbour given by its pair-table offset
__device__ __forceinline__ int cross_index_of_lin(const Geom &g, int lin)
{
    const long long i = g.pair_center + lin;
    const int dx = (int)(i % g.pnx) - g.phx, dy = (int)((i / g.pnx) % g.pny) - g.phy,
              dz = (int)(i / ((long long)g.pnx * g.pny)) - g.phz;
    return ((dz + g.rz) * (2 * g.ry + 1) + (dy + g.ry)) * (2 * g.rx + 1) + (dx + g.rx);
}

// the reference's fallback and combine, on the target's values
__device__ __forceinline__ void cok_write(const CokArgsDev &a, int cell, int status, float result, float sv)
{
    if (status != 0) result = __fsub_rn(__fadd_rn(a.p.pm, sv), a.p.sm); // pm + sv - sm in float
    a.out_data[cell] = result;
    a.out_mask[cell] = 1;
    if (a.status) a.status[cell] = (signed char)status;
}

// n <= 32: a target per warp on the FP64 tensor instruction (warp64.cuh), b and
// the cross covariances as its two right-hand sides. 20 warps of 96 registers an
// SM; two targets per warp in folded rows, 8 warps an SM, took 12.3 ms for the
// 1.82M targets of a 160x144x80 grid with 32 neighbours; this takes 7.8.
constexpr int kCokThreads = 640;

__global__ void __launch_bounds__(kCokThreads, 1) k_cok_solve_warp(const CokArgsDev a)
{
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    WarpSmem<2, false> &T = reinterpret_cast<WarpSmem<2, false> *>(smem)[threadIdx.x >> 5];
    const Geom &g = a.g;
    const double *pair_c = a.pair64 + g.pair_center;
    const int stride = gridDim.x * (kCokThreads / 32);
    // the next target's record is loaded during the current solve
    int it = blockIdx.x * (kCokThreads / 32) + (threadIdx.x >> 5);
    int cell = 0, n = 0, ncell = 0, nn = 0;
    int2 rec = make_int2(0, 0);
    auto load = [&](int c, int m) { return lane < m ? a.nb_rec[(long long)c * a.k + lane] : make_int2(0, 0); };
    if (it < a.n_targets)
    {
        cell = a.targets[it];
        n = a.nb_n[cell];
        rec = load(cell, n);
    }
    if (it + stride < a.n_targets) ncell = a.targets[it + stride];
    for (; it < a.n_targets; it += stride)
    {
        const int lin = rec.x;
        double b = 0.0, c = 0.0;
        if (lane < n)
        {
            b = __ldg(pair_c + abs(lin));
            c = __dmul_rn(a.p.coef, a.cross_tab[cross_index_of_lin(g, lin)]);
        }
        const float v = __int_as_float(rec.y);
        const float sv = a.smask[cell] ? a.sdata[cell] : a.p.sm;
        T.lin[lane] = lin;
        T.y[0][lane] = b;
        T.y[1][lane] = c;
        __syncwarp();
        const int nb = (n + 7) >> 3;
        nn = it + stride < a.n_targets ? a.nb_n[ncell] : 0;
        const bool fail = warp_factor<2, true, false, true>(T, lane, n, nb, pair_c);
        rec = load(ncell, nn);
        warp_back<2>(T, lane, nb);
        const double x = lane < n ? T.y[0][lane] : 0.0, y = lane < n ? T.y[1][lane] : 0.0;
        // the border: wn = (b_n - c.x) / (s - c.y)
        double cx = c * x, cy = c * y;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            cx += __shfl_xor_sync(FULL, cx, o);
            cy += __shfl_xor_sync(FULL, cy, o);
        }
        const double piv = a.p.sec_var - cy;
        const bool bad = fail || !(fabs(piv) >= DBL_EPSILON);
        const double wn = bad ? 0.0 : (a.p.b_last - cx) / piv;
        // combine: result accumulated in double per term, stored as float
        __syncwarp();
        T.y[0][lane] = __dmul_rn((double)__fsub_rn(v, a.p.pm), __dsub_rn(x, __dmul_rn(wn, y)));
        __syncwarp();
        float result = a.p.pm;
#pragma unroll 4
        for (int i = 0; i < n; ++i) result = __double2float_rn(__dadd_rn((double)result, T.y[0][i]));
        result = __double2float_rn(__dadd_rn((double)result, __dmul_rn(wn, (double)__fsub_rn(sv, a.p.sm))));
        if (lane == 0) cok_write(a, cell, n == 0 ? 1 : (bad ? 2 : 0), result, sv);
        cell = ncell;
        n = nn;
        ncell = it + 2 * stride < a.n_targets ? a.targets[it + 2 * stride] : 0;
        __syncwarp();
    }
}

// 32 < n <= kSgsBlockMax: one block per target, A in shared memory.
constexpr int kCokBlockThreads = 128;

__global__ void __launch_bounds__(kCokBlockThreads) k_cok_solve_block(const CokArgsDev a)
{
    extern __shared__ double sh[];
    const int kk = a.k;
    double *A = sh;                  // kk * kk
    double *b = A + (size_t)kk * kk; // b
    double *c = b + kk;              // cross covariances
    double *x = c + kk;              // A^-1 b
    double *y = x + kk;              // A^-1 c
    float *vals = reinterpret_cast<float *>(y + kk);
    __shared__ int s_fail;
    const Geom &g = a.g;
    const long long pc = g.pair_center;
    for (int it = blockIdx.x; it < a.n_targets; it += gridDim.x)
    {
        const int cell = a.targets[it];
        const int n = a.nb_n[cell];
        const int2 *row = a.nb_rec + (long long)cell * kk;
        for (int e = threadIdx.x; e < n * n; e += blockDim.x)
        {
            const int i = e / n, j = e % n;
            A[(size_t)i * n + j] = a.pair64[pc + row[i].x - row[j].x];
        }
        for (int i = threadIdx.x; i < n; i += blockDim.x)
        {
            const int2 rec = row[i];
            b[i] = a.pair64[pc + rec.x];
            c[i] = __dmul_rn(a.p.coef, a.cross_tab[cross_index_of_lin(g, rec.x)]);
            vals[i] = __int_as_float(rec.y);
        }
        if (threadIdx.x == 0) s_fail = 0;
        __syncthreads();
        for (int j = 0; j < n; ++j)
        {
            const double d = A[(size_t)j * n + j];
            if (threadIdx.x == 0 && !(d >= DBL_EPSILON)) s_fail = 1;
            const double ljj = sqrt(d);
            __syncthreads();
            for (int i = j + 1 + threadIdx.x; i < n; i += blockDim.x) A[(size_t)i * n + j] /= ljj;
            if (threadIdx.x == 0) A[(size_t)j * n + j] = ljj;
            __syncthreads();
            const int span = n - j - 1;
            for (int e = threadIdx.x; e < span * span; e += blockDim.x)
            {
                const int i = j + 1 + e / span, cc = j + 1 + e % span;
                if (cc <= i) A[(size_t)i * n + cc] -= A[(size_t)i * n + j] * A[(size_t)cc * n + j];
            }
            __syncthreads();
        }
        if (threadIdx.x < 2)
        {
            double *xv = threadIdx.x == 0 ? x : y;
            const double *src = threadIdx.x == 0 ? b : c;
            for (int i = 0; i < n; ++i)
            {
                double s = src[i];
                for (int q = 0; q < i; ++q) s -= A[(size_t)i * n + q] * xv[q];
                xv[i] = s / A[(size_t)i * n + i];
            }
            for (int i = n - 1; i >= 0; --i)
            {
                double s = xv[i];
                for (int q = i + 1; q < n; ++q) s -= A[(size_t)q * n + i] * xv[q];
                xv[i] = s / A[(size_t)i * n + i];
            }
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            const float sv = a.smask[cell] ? a.sdata[cell] : a.p.sm;
            int status = 1;
            float result = 0.0f;
            if (n > 0)
            {
                double cxs = 0.0, cys = 0.0;
                for (int i = 0; i < n; ++i)
                {
                    cxs += c[i] * x[i];
                    cys += c[i] * y[i];
                }
                const double piv = a.p.sec_var - cys;
                const bool bad = s_fail || !(fabs(piv) >= DBL_EPSILON);
                const double wn = bad ? 0.0 : (a.p.b_last - cxs) / piv;
                result = a.p.pm;
                for (int i = 0; i < n; ++i)
                    result = __double2float_rn(__dadd_rn(
                        (double)result,
                        __dmul_rn((double)__fsub_rn(vals[i], a.p.pm), __dsub_rn(x[i], __dmul_rn(wn, y[i])))));
                result = __double2float_rn(__dadd_rn((double)result, __dmul_rn(wn, (double)__fsub_rn(sv, a.p.sm))));
                status = bad ? 2 : 0;
            }
            cok_write(a, cell, status, result, sv);
        }
        __syncthreads();
    }
}

void launch_cok_prepare(long long n, const uint8_t *pmask, int *flag, cudaStream_t st)
{
    k_cok_prepare<<<1184, 256, 0, st>>>(n, pmask, flag);
}
void launch_cok_targets(long long n, const int *flag, const int *pos, int *targets, cudaStream_t st)
{
    k_cok_targets<<<1184, 256, 0, st>>>(n, flag, pos, targets);
}
void launch_cok_finalize(long long n, const float *pdata, const uint8_t *pmask, float *out_data, uint8_t *out_mask,
                         signed char *status, cudaStream_t st)
{
    k_cok_finalize<<<1184, 256, 0, st>>>(n, pdata, pmask, out_data, out_mask, status);
}

cudaError_t launch_cok_solve(const Geom &g, const int *targets, int n_targets, const int2 *nb_rec, const int *nb_n,
                             int k, const double *pair64, const double *cross_tab, const float *pdata,
                             const float *sdata, const uint8_t *smask, const CokParams &p, float *out_data,
                             uint8_t *out_mask, signed char *status, int n_sm, cudaStream_t st)
{
    if (n_targets <= 0) return cudaSuccess;
    CokArgsDev a{g, targets, n_targets, nb_rec, nb_n, k, pair64, cross_tab, pdata, sdata, smask, p, out_data, out_mask,
                 status};
    if (k <= 32)
    {
        constexpr int warps = kCokThreads / 32;
        const size_t smem = sizeof(WarpSmem<2, false>) * warps;
        int per_sm = 0;
        cudaError_t e = set_smem_min_carveout(k_cok_solve_warp, kCokThreads, smem, per_sm);
        if (e != cudaSuccess) return e;
        k_cok_solve_warp<<<std::min((n_targets + warps - 1) / warps, n_sm), kCokThreads, smem, st>>>(a);
    }
    else
    {
        const size_t smem = (size_t)k * k * 8 + 4 * (size_t)k * 8 + (size_t)k * 4;
        cudaError_t e = cudaFuncSetAttribute(k_cok_solve_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        const int blocks = std::min(n_targets, n_sm * 8);
        k_cok_solve_block<<<blocks, kCokBlockThreads, smem, st>>>(a);
    }
    return cudaGetLastError();
}
} // namespace hb
