// The kriging weights of sequential simulation, solved ahead of the levels.
//
// A node's weights and variance depend on where its neighbours are, not on
// their simulated values, so the solves need not wait for one another: one
// launch solves the systems of every node (of a chunk of them, in level order),
// and a level is left with sums over stored weights and the draw. Solved level
// by level (434 launches on the 200x200x100 SIS grid), each level ended in a
// part-filled wave of 8-warp blocks.
//
// Stored per chunk, by position in level order and category: kmax weights W, the
// neighbour count and status, and SGS's variance.
#include "engine.cuh"
#include "kernels.h"
#include "sim_common.cuh"
#include "warp64.cuh"

#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

namespace hb
{
// 20 warps of 96 registers (the chain of pivots is what a warp waits for)
constexpr int kWeightThreads = 640;

__device__ __forceinline__ int fast_div(int x, const FastDiv &f)
{
    return f.s ? (int)(__umulhi((unsigned)x, f.m) >> (f.s - 1)) : x;
}

enum SimMode
{
    kSimSK = 0,  // SGS, simple kriging
    kSimOK = 1,  // SGS, ordinary kriging
    kSimIK = 2,  // SIS
    kSimCorr = 3 // SIS, correlogram weights: A_ij = C_ij (s_i s_j), b_i = C_ic (s_i s_c)
};

template <int MODE>
__global__ void __launch_bounds__(kWeightThreads, 1) k_sim_weights(const SimWeights a)
{
    constexpr int Q = MODE == kSimOK ? 2 : 1;
    constexpr bool CORR = MODE == kSimCorr, SGS = MODE <= kSimOK;
    typedef WarpSmem<Q, CORR> Smem;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    Smem &T = reinterpret_cast<Smem *>(smem)[threadIdx.x >> 5];
    const int n_sys = a.count * a.kcat; // category after category
    const int stride = gridDim.x * (kWeightThreads / 32);
    // the next system's chain of dependent loads (rank; count; neighbours)
    // is issued a stage at a time during the current solve
    struct Item
    {
        int cat, pos, r, n, cell, q; // q: the lane's neighbour (the node itself beyond n)
    };
    auto stage_a = [&](int it, Item &s) {
        s.cat = 0;
        s.pos = 0;
        s.r = -1;
        if (it < n_sys)
        {
            s.cat = a.kcat > 1 ? it / a.count : 0;
            s.pos = it - s.cat * a.count;
            s.r = a.order[a.first + s.pos];
        }
    };
    auto stage_b = [&](Item &s) {
        s.n = s.r >= 0 ? __ldg(a.cats[s.cat].nb_cnt + s.r) : 0;
        s.cell = s.r >= 0 ? __ldg(a.sim_cells + s.r) : 0;
    };
    auto stage_c = [&](Item &s) {
        const SisCat &C = a.cats[s.cat];
        s.q = lane < s.n ? __ldg(C.nb + (long long)s.r * C.k + lane) : s.cell;
    };
    int it = blockIdx.x * (kWeightThreads / 32) + (threadIdx.x >> 5);
    Item cur, nxt;
    stage_a(it, cur);
    stage_b(cur);
    stage_c(cur);
    stage_a(it + stride, nxt);
    for (; it < n_sys; it += stride)
    {
        const SisCat &C = a.cats[cur.cat];
        const double *pair_c = C.pair64 + C.pair_center;
        const int n = cur.n;
        // ---- this warp's system. The neighbours' pair-table offsets are formed here:
        // stored by the search they took four bytes more a neighbour
        const int rows_q = fast_div(cur.q, a.nx), rows_c = fast_div(cur.cell, a.nx);
        const int z_q = fast_div(rows_q, a.ny), z_c = fast_div(rows_c, a.ny);
        const int dz = z_q - z_c, dy = rows_q - rows_c - (int)a.ny.d * dz;
        const int dx = cur.q - cur.cell - (int)a.nx.d * (rows_q - rows_c);
        const int lin = dx + C.pnx * (dy + C.pny * dz);
        double bi = 0.0;
        {
            double s = 1.0;
            if (lane < n)
            {
                bi = __ldg(pair_c + abs(lin));
                if (CORR)
                {
                    s = sis_sigma(C.means ? C.means[cur.q] : C.marginal);
                    bi = __dmul_rn(bi, __dmul_rn(s, sis_sigma(C.means ? C.means[cur.cell] : C.marginal)));
                }
            }
            T.lin[lane] = lin;
            T.y[0][lane] = bi;
            if (Q == 2) T.y[Q - 1][lane] = lane < n ? 1.0 : 0.0;
            if (CORR) T.sig[lane] = s;
        }
        __syncwarp();
        const int nb = (n + 7) >> 3;
        stage_b(nxt);
        const bool fail = warp_factor<Q, false, CORR>(T, lane, n, nb, pair_c);
        stage_c(nxt);
        warp_back<Q>(T, lane, nb);

        // ---- lane i: weight i, and the sums in the neighbours' order (what is
        // beyond n is zero and changes none)
        int status = n == 0 ? 1 : (fail ? 2 : 0);
        double x = lane < n ? T.y[0][lane] : 0.0, mu = 0.0;
        if constexpr (MODE == kSimOK)
        {
            double sx = 0.0, sy = 0.0;
#pragma unroll 4
            for (int i = 0; i < 8 * nb; i += 2)
            {
                const double2 u = *reinterpret_cast<const double2 *>(&T.y[0][i]);
                const double2 v = *reinterpret_cast<const double2 *>(&T.y[1][i]);
                sx = __dadd_rn(__dadd_rn(sx, u.x), u.y);
                sy = __dadd_rn(__dadd_rn(sy, v.x), v.y);
            }
            const bool bad = fabs(sy) < 1e-15;
            if (bad && n > 0) status = 2;
            mu = bad ? 0.0 : __ddiv_rn(__dsub_rn(sx, 1.0), sy);
            x = __dsub_rn(x, __dmul_rn(mu, lane < n ? T.y[Q - 1][lane] : 0.0));
        }
        const long long at = ((long long)cur.pos * a.kcat + cur.cat) * a.kmax + lane;
        if (lane < n)
            a.W[at] = x;
        if constexpr (SGS)
        {
            __syncwarp();
            T.y[0][lane] = __dmul_rn(x, bi);
            __syncwarp();
            double var = __ldg(pair_c);
#pragma unroll 4
            for (int i = 0; i < 8 * nb; i += 2)
            {
                const double2 v = *reinterpret_cast<const double2 *>(&T.y[0][i]);
                var = __dsub_rn(__dsub_rn(var, v.x), v.y);
            }
            if (MODE == kSimOK) var = __dsub_rn(var, mu);
            if (var < 0) var = 0;
            if (lane == 0) a.var[cur.pos] = var;
        }
        if (lane == 0)
        {
            a.n[(long long)cur.pos * a.kcat + cur.cat] = (unsigned char)n;
            a.st[(long long)cur.pos * a.kcat + cur.cat] = (signed char)status;
        }
        cur = nxt;
        stage_a(it + 2 * stride, nxt);
        __syncwarp();
    }
}

// ------------------------------------------------------------------ levels
// Blocks of 32 (node, category) rows: a warp forms a row's terms, weight times
// value, lane i the i-th, then one lane a row sums them in the neighbours' order
// (values of lower levels are final). The rows of a node are stored together:
// position-major rows of one neighbour each, which one thread a node would read
// coalesced, lie megabytes apart and took 33 us a level in TLB misses.
//
// A level is a few thousand nodes: what it takes is the chain of its loads (order,
// neighbours, values, then the sums and the draw) and the launch. All but the
// values are there before the level below is done, so a level is launched as soon
// as the blocks of the one below have started (programmatic dependent launch),
// reads what is there, and waits for the values (read past L1, which blocks of the
// level below share). Every thread waits, so a level ends after the one below.
// 364 levels of 8.3M nodes: 4.5 -> 2.1 ms; 426 levels of 4M nodes with five
// categories: 2.1 ms less.
constexpr int kLevelRows = 32, kLevelWarps = 8, kLevelPer = kLevelRows / kLevelWarps;

__device__ __forceinline__ void level_started() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void level_below_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__global__ void __launch_bounds__(32 * kLevelWarps) k_sgs_level(
    const SimWeights a, int first, int count, float *__restrict__ data, const float *__restrict__ means,
    const double *__restrict__ uniforms, signed char *__restrict__ st_rank)
{
    __shared__ float term[kLevelRows][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row0 = blockIdx.x * kLevelRows;
    level_started();
    int q[kLevelPer];
    double w[kLevelPer];
#pragma unroll
    for (int e = 0; e < kLevelPer; ++e)
    {
        const int j = warp + e * kLevelWarps, pos = first + row0 + j;
        q[e] = -1;
        if (row0 + j < count && lane < a.n[pos])
        {
            q[e] = a.cats[0].nb[(long long)a.order[a.first + pos] * a.kmax + lane];
            w[e] = a.W[(long long)pos * a.kmax + lane];
        }
    }
    const bool mine = warp == 0 && row0 + lane < count;
    int r = 0, cell = 0, n = 0, status = 0;
    double u = 0.0, var = 0.0;
    if (mine)
    {
        const int pos = first + row0 + lane;
        r = a.order[a.first + pos];
        cell = a.sim_cells[r];
        n = a.n[pos];
        status = a.st[pos];
        u = uniforms[r];
        var = a.var[pos];
    }
    level_below_done();
#pragma unroll
    for (int e = 0; e < kLevelPer; ++e)
    {
        float t = 0.0f;
        if (q[e] >= 0)
        {
            const float d = __ldcg(data + q[e]), v = means ? __fsub_rn(d, means[q[e]]) : d;
            t = __double2float_rn(__dmul_rn(w[e], (double)v));
        }
        term[warp + e * kLevelWarps][lane] = t;
    }
    __syncthreads();
    if (!mine) return;
    float est = means ? means[cell] : 0.0f;
#pragma unroll 8
    for (int i = 0; i < n; ++i) est = __fadd_rn(est, term[lane][i]);
    const double val = status == 0 ? sgs_gauss_inverse(u, (double)est, var) : sgs_gauss_inverse(u, 0.0, 1.0);
    data[cell] = __double2float_rn(val);
    st_rank[r] = (signed char)status;
}

// SIS: 32 / kcat nodes a block, each with its kcat rows, then the picks.
__global__ void __launch_bounds__(32 * kLevelWarps) k_sis_level(
    const SimWeights a, int first, int count, int ncat, uint8_t *__restrict__ data,
    const double *__restrict__ uniforms, signed char *__restrict__ st_rank)
{
    __shared__ double term[kLevelRows][33];
    __shared__ double prob[kLevelRows];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nodes = kLevelRows / a.kcat, rows = nodes * a.kcat;
    const int node0 = blockIdx.x * nodes;
    level_started();
    int q[kLevelPer];
    double w[kLevelPer];
    float mean[kLevelPer];
#pragma unroll
    for (int e = 0; e < kLevelPer; ++e)
    {
        const int j = warp + e * kLevelWarps, cat = j % a.kcat, node = node0 + j / a.kcat;
        const long long row = (long long)(first + node) * a.kcat + cat;
        q[e] = -1;
        if (j < rows && node < count && lane < a.n[row])
        {
            const SisCat &C = a.cats[cat];
            q[e] = C.nb[(long long)a.order[a.first + first + node] * C.k + lane];
            w[e] = a.W[row * a.kmax + lane];
            mean[e] = C.means ? C.means[q[e]] : C.marginal;
        }
    }
    level_below_done();
#pragma unroll
    for (int e = 0; e < kLevelPer; ++e)
    {
        const int j = warp + e * kLevelWarps;
        if (j >= rows) break;
        double t = 0.0;
        // indicator - mean, in float
        if (q[e] >= 0) t = __dmul_rn(w[e], (double)__fsub_rn(__ldcg(data + q[e]) == j % a.kcat ? 1.0f : 0.0f, mean[e]));
        term[j][lane] = t;
    }
    __syncthreads();
    if (warp != 0) return;
    if (lane < rows && node0 + lane / a.kcat < count)
    {
        const int cat = lane % a.kcat, pos = first + node0 + lane / a.kcat;
        const long long row = (long long)pos * a.kcat + cat;
        const SisCat &C = a.cats[cat];
        const double mc = (double)(C.means ? C.means[a.sim_cells[a.order[a.first + pos]]] : C.marginal);
        const int n = a.n[row];
        double p = mc;
#pragma unroll 8
        for (int i = 0; i < n; ++i) p = __dadd_rn(p, term[lane][i]);
        prob[lane] = a.st[row] == 0 ? p : mc;
    }
    __syncwarp();
    if (lane >= nodes || node0 + lane >= count) return;
    // the sum, then the first category whose running sum exceeds u times it
    const int pos = first + node0 + lane;
    const int r = a.order[a.first + pos], cell = a.sim_cells[r];
    const double *p = prob + lane * a.kcat;
    const double p0 = p[0];
    double sum = 0.0;
    int stv = 0;
    for (int c = 0; c < a.kcat; ++c)
    {
        sum = __dadd_rn(sum, p[c]);
        stv = max(stv, (int)a.st[(long long)pos * a.kcat + c]);
    }
    if (ncat == 2) sum = __dadd_rn(sum, __dsub_rn(1.0, p0)); // median SIS: p1 = 1 - p0
    const double s = __dmul_rn(uniforms[r], sum);
    double acc = 0.0;
    int pick = ncat - 1;
    for (int c = 0; c < ncat; ++c)
    {
        acc = __dadd_rn(acc, ncat == 2 && c == 1 ? __dsub_rn(1.0, p0) : p[c]);
        if (s < acc)
        {
            pick = c;
            break;
        }
    }
    data[cell] = (uint8_t)pick;
    st_rank[r] = (signed char)stv;
}

// ------------------------------------------------------------------ launchers
template <int MODE>
static cudaError_t launch_weights(const SimWeights &a, int n_sm, cudaStream_t st)
{
    constexpr int warps = kWeightThreads / 32;
    const size_t smem = sizeof(WarpSmem<MODE == kSimOK ? 2 : 1, MODE == kSimCorr>) * warps;
    auto kern = k_sim_weights<MODE>;
    int per_sm = 0;
    const cudaError_t e = set_smem_min_carveout(kern, kWeightThreads, smem, per_sm);
    if (e != cudaSuccess) return e;
    const int n_sys = a.count * a.kcat;
    kern<<<std::max(1, std::min((n_sys + warps - 1) / warps, n_sm)), kWeightThreads, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sim_weights(const SimWeights &a, bool sgs, bool ordinary, bool correlogram, int n_sm,
                               cudaStream_t st)
{
    if (a.count <= 0) return cudaSuccess;
    if (sgs) return ordinary ? launch_weights<kSimOK>(a, n_sm, st) : launch_weights<kSimSK>(a, n_sm, st);
    return correlogram ? launch_weights<kSimCorr>(a, n_sm, st) : launch_weights<kSimIK>(a, n_sm, st);
}

// beside: the launch before this one in the stream is the level below
template <typename... P, typename... A>
static cudaError_t launch_level(void (*kern)(P...), int blocks, bool beside, cudaStream_t st, A... args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(32 * kLevelWarps);
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = beside ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
    if (e == cudaErrorNotSupported && beside)
    {
        // a stream that does not take the attribute: one level after another
        cudaGetLastError();
        cfg.numAttrs = 0;
        e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
    }
    return e;
}

cudaError_t launch_sgs_level(const SimWeights &a, int first, int count, bool beside, float *data, const float *means,
                             const double *uniforms, signed char *st_rank, cudaStream_t st)
{
    if (count <= 0) return cudaSuccess;
    return launch_level(k_sgs_level, (count + kLevelRows - 1) / kLevelRows, beside, st, a, first, count, data, means,
                        uniforms, st_rank);
}

cudaError_t launch_sis_level(const SimWeights &a, int first, int count, bool beside, int ncat, uint8_t *data,
                             const double *uniforms, signed char *st_rank, cudaStream_t st)
{
    if (count <= 0) return cudaSuccess;
    const int nodes = kLevelRows / a.kcat;
    return launch_level(k_sis_level, (count + nodes - 1) / nodes, beside, st, a, first, count, ncat, data, uniforms,
                        st_rank);
}
} // namespace hb
