// FP64 kriging solves on the FP64 tensor instruction: one system per warp
// (mma64.cuh), for every neighbour-count bucket up to 64.
#include "engine.cuh"
#include "kernels.h"
#include "mma64.cuh"
#include "solve_common.cuh"

#include <cstdint>
#include <cuda_runtime.h>

namespace hb
{
// shared memory of one system: the rows b, 1 and v - mean, the pair-table
// offsets of the unknowns
template <int NB>
struct MmaSmem
{
    static constexpr int N = 8 * NB;
    static constexpr int doubles = 3 * N + N / 2;
};

template <int NB, bool ORDINARY, int TH>
__global__ void __launch_bounds__(TH, 1)
    k_solve_mma(const Geom g, const int2 *__restrict__ cells, const int *__restrict__ n_items_ptr,
                const int2 *__restrict__ nb_rec, int ind_value, SolveParams P)
{
    constexpr int N = 8 * NB;
    constexpr int RPL = N / 32; // records per lane
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int r = lane >> 2, q = lane & 3;
    double *xs = reinterpret_cast<double *>(smem) + (size_t)warp * (MmaSmem<NB>::doubles + kMmaRowDoubles);
    int *lin = reinterpret_cast<int *>(xs + 3 * N);
    double *row = xs + MmaSmem<NB>::doubles;
    const double *pair_c = P.pair64 + P.pc;

    const int n_items = *n_items_ptr;
    const int per_block = (n_items + gridDim.x - 1) / gridDim.x;
    const int run_first = blockIdx.x * per_block;
    const int run_end = min(n_items, run_first + per_block);
    int it = run_first + warp;
    // the records of the next system are loaded during the current one
    int2 w_cur = it < run_end ? cells[it] : make_int2(0, 0);
    int2 w_nxt = it + nwarps < run_end ? cells[it + nwarps] : make_int2(0, 0);
    int2 rec[RPL];
    auto load_rec = [&](const int2 &w) {
#pragma unroll
        for (int e = 0; e < RPL; ++e)
        {
            const int i = lane + 32 * e;
            rec[e] = i < w.y ? nb_rec[(long long)w.x * g.k + i] : make_int2(0, 0);
        }
    };
    load_rec(w_cur);
    for (; it < run_end; it += nwarps)
    {
        const int cell = w_cur.x, n = w_cur.y, nb = (n + 7) >> 3;
#pragma unroll
        for (int e = 0; e < RPL; ++e)
        {
            const int i = lane + 32 * e, at = mma_slot(i, n, nb);
            const bool live = i < n;
            lin[at] = rec[e].x;
            xs[at] = live ? __ldg(pair_c + abs(rec[e].x)) : 0.0;
            if (ORDINARY) xs[N + at] = live ? 1.0 : 0.0;
            xs[2 * N + at] = centred_value(live, __int_as_float(rec[e].y), ind_value, P.mf);
        }
        __syncwarp();
        Blk A[NB * (NB + 1) / 2], X[NB];
        bool fail = false;
        mma_load<NB>(A, pair_c, lin, n, nb, lane);
        const bool used = ORDINARY ? r < 3 : (r == 0 || r == 2);
#pragma unroll
        for (int k = 0; k < NB; ++k)
        {
            double2 v = make_double2(0.0, 0.0);
            if (used) v = reinterpret_cast<const double2 *>(xs + r * N + 8 * k)[q];
            X[k] = Blk{v.x, v.y};
        }
        load_rec(w_nxt);
        w_cur = w_nxt;
        w_nxt = it + 2 * nwarps < run_end ? cells[it + 2 * nwarps] : make_int2(0, 0);
        half_factor<NB, true, false, false>(A, X, nb, row, lane, fail);
        Blk G{0.0, 0.0};
#pragma unroll
        for (int k = 0; k < NB; ++k)
            if (k < nb) blk_mul_t(G, X[k], X[k]);
        // rows 0 = b, 1 = ones, 2 = v - mean: lane 0 has (0,0) and (0,1)
        const double s_vb = __shfl_sync(0xffffffffu, G.x, 1);
        double s_11 = 0.0, s_v1 = 0.0;
        if (ORDINARY)
        {
            s_11 = __shfl_sync(0xffffffffu, G.y, 4);
            s_v1 = __shfl_sync(0xffffffffu, G.x, 5);
        }
        if (lane == 0) write_solution<ORDINARY>(P, cell, fail, s_vb, G.x, G.y, s_v1, s_11);
        __syncwarp();
    }
}

template <int NB, bool ORD, int TH>
static cudaError_t launch_mma(const Geom &g, const int2 *cells, const int *n_items, int max_items, const int2 *nb_rec,
                              int ind_value, const SolveParams &P, int n_sm, cudaStream_t st)
{
    const size_t smem = (size_t)(TH / 32) * (MmaSmem<NB>::doubles + kMmaRowDoubles) * sizeof(double);
    auto kern = k_solve_mma<NB, ORD, TH>;
    int blocks = 0;
    cudaError_t e = launch_kernel(kern, TH, smem, max_items, TH / 32, n_sm, blocks);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)blocks, TH, smem, st>>>(g, cells, n_items, nb_rec, ind_value, P);
    return cudaGetLastError();
}

// Buckets of 17 to 32 and of 33 to 64 neighbours (smaller ones are faster in
// the folded kernel). 640 threads at 96 registers with a few spills beat 512
// without (20.5 against 21.8 ms for 8.3M systems of 32): the chain of 32
// pivots is what a warp waits for, so more of them in flight pay.
cudaError_t launch_solve_mma(int np, bool ordinary, const Geom &g, const int2 *cells, const int *n_items,
                             int max_items, const int2 *nb_rec, int ind_value, const SolveParams &P, int n_sm,
                             cudaStream_t st)
{
#define HB_ARGS g, cells, n_items, max_items, nb_rec, ind_value, P, n_sm, st
    if (np == 32) return ordinary ? launch_mma<4, true, 640>(HB_ARGS) : launch_mma<4, false, 640>(HB_ARGS);
    if (np == 64) return ordinary ? launch_mma<8, true, 256>(HB_ARGS) : launch_mma<8, false, 256>(HB_ARGS);
    return cudaErrorInvalidValue;
#undef HB_ARGS
}
} // namespace hb
