// FP64 kriging solves that share one factorisation between neighbouring cells.
//
// Cells next to each other have almost the same neighbours: moving one cell
// along x changes one or two of 32 at the benchmark's density. A warp takes up
// to eight such cells of a bucket's list, finds the neighbours
// that all of them have, and orders every cell's system with 8 cb of those
// first (cb = ceil(n / 8) - 1) and the cell's remaining at most eight
// neighbours, its extras, last. Then
//   * the common block is assembled and factored once (mma64.cuh, tensor FP64),
//   * every distinct extra, every cell's right-hand side b, the ones and the
//     values v - mean are forward-substituted through it once, as rows of one
//     matrix R in shared memory,
//   * a cell adds only its own Schur complement S = A_EE - R_E R_E^T (8x8) with
//     the right-hand sides X_E - X R_E^T, and the elimination of S, four cells
//     at a time on eight lanes each.
// Each cell still solves its own whole system, in another order of unknowns.
// Groups come from tiles of eight cells (the list is in tile order), the
// largest of 8, 4, 2 following cells with 8 cb common neighbours; cells that
// share with no other go to a queue (left_cells) for
// the one-system-per-warp kernel, and so does a cell with a failing pivot (which the
// cell's own order of unknowns may not have).
#include "engine.cuh"
#include "kernels.h"
#include "mma64.cuh"
#include "solve_common.cuh"

#include <cstdint>
#include <cuda_runtime.h>

namespace hb
{
constexpr int kShareRows = 32; // rows of R: extras, b's, ones, values
constexpr int kShareCells = 8; // cells of a group at most
constexpr int kShareEmpty = (int)0x80000000;

template <int CB>
struct ShareCfg
{
    static constexpr int N = 8 * CB + 8;           // largest neighbour count
    static constexpr int RPL = (N + 31) / 32;      // records per lane and cell
    static constexpr int T = RPL == 1 ? 128 : 256; // hash slots
    static constexpr int LD = 8 * CB;              // row length of R
};

template <int CB>
struct __align__(16) ShareWarp
{
    typedef ShareCfg<CB> K;
    double R[kShareRows * K::LD];
    union
    {
        struct // the neighbours of the window's cells, by hash of their offset
        {
            int key[K::T];
            int mask[K::T]; // bit c: neighbour of cell c
            float val[K::T];
        };
        struct
        {
            double S[4][64];     // Schur complements (16-byte chunks swizzled)
            double XE[4][3 * 8]; // their right-hand sides
        };
    };
    double row[2 * 4 * 12];    // broadcast rows of the eliminations (and of mma_diag)
    double F[kShareCells][6];  // forms per cell, a failed pivot
    int clin[K::LD];           // common neighbours: offsets, values
    float cval[K::LD];
    int rlin[kShareRows];      // rows of R: offsets, values
    float rval[kShareRows];
    unsigned char id[K::T];    // slot -> row of R, 255 common
    unsigned char slot[kShareCells][32 * K::RPL]; // neighbour -> slot
    unsigned char eid[kShareCells][8];            // extra -> row of R
};

template <int CB, bool ORDINARY, int TH, bool HALVES>
__global__ void __launch_bounds__(TH, 1)
    k_solve_share(const Geom g, const int2 *__restrict__ cells, const int *__restrict__ n_items_ptr,
                  const int2 *__restrict__ nb_rec, int ind_value, SolveParams P, CellTile tile,
                  int2 *__restrict__ left_cells, int *__restrict__ left_count)
{
    typedef ShareCfg<CB> K;
    constexpr int RPL = K::RPL, W = kShareCells, T = K::T, LD = K::LD;
    constexpr int Q = ORDINARY ? 3 : 2; // right-hand sides: b, (1,) v - mean
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r = lane >> 2, q = lane & 3;
    ShareWarp<CB> &sh = reinterpret_cast<ShareWarp<CB> *>(smem)[warp];
    const double *pair_c = P.pair64 + P.pc;
    const unsigned below = (1u << lane) - 1u;

    // a contiguous run of the list per warp, a multiple of the window
    const int n_items = *n_items_ptr;
    const int n_warps = gridDim.x * (TH / 32);
    const int chunk = ((n_items + n_warps - 1) / n_warps + W - 1) / W * W;
    const long long first = (long long)(blockIdx.x * (TH / 32) + warp) * chunk;
    const int run_end = (int)min((long long)n_items, first + chunk);
    for (int base = (int)min(first, (long long)n_items); base < run_end;)
    {
        // ---- the window: the following list entries in the same tile
        int2 my = make_int2(0, 0);
        if (lane < W && base + lane < run_end) my = cells[base + lane];
        int my_off, w; // offset of the lane's cell from the first one's
        {
            const int x = my.x % g.nx, y = my.x / g.nx % g.ny, z = my.x / g.nx / g.ny;
            const int x0 = __shfl_sync(FULL, x, 0), y0 = __shfl_sync(FULL, y, 0), z0 = __shfl_sync(FULL, z, 0);
            const bool in = lane < W && base + lane < run_end && x >> tile.lx == x0 >> tile.lx &&
                            y >> tile.ly == y0 >> tile.ly && z >> tile.lz == z0 >> tile.lz;
            w = __ffs(~__ballot_sync(FULL, in)) - 1;
            my_off = pair_lin(g, x - x0, y - y0, z - z0);
        }
        for (int i = lane; i < T; i += 32)
        {
            sh.key[i] = kShareEmpty;
            sh.mask[i] = 0;
        }
        __syncwarp();
        // ---- which cells have which neighbour: open addressing
        bool over = false;
        auto load = [&](int c, int2 (&rec)[RPL]) { // the lane's records of cell c, none from w on
            const int cell = __shfl_sync(FULL, my.x, c), n = __shfl_sync(FULL, my.y, c);
#pragma unroll
            for (int e = 0; e < RPL; ++e)
            {
                const int i = lane + 32 * e;
                rec[e] = c < w && i < n ? nb_rec[(long long)cell * g.k + i] : make_int2(kShareEmpty, 0);
            }
        };
        auto insert = [&](int c, const int2 (&rec)[RPL]) {
            const int off = __shfl_sync(FULL, my_off, c);
#pragma unroll
            for (int e = 0; e < RPL; ++e)
                if (rec[e].x != kShareEmpty)
                {
                    const int key = rec[e].x + off;
                    int s = (int)(((unsigned)key * 0x9E3779B1u) >> 16) & (T - 1);
                    int tries = 0;
                    for (; tries < 32; ++tries)
                    {
                        const int old = atomicCAS(&sh.key[s], kShareEmpty, key);
                        if (old == kShareEmpty || old == key) break;
                        s = (s + 1) & (T - 1);
                    }
                    if (tries == 32) over = true;
                    else
                    {
                        const float v = __int_as_float(rec[e].y);
                        sh.val[s] = (ind_value >= 0 ? (v == (float)ind_value ? 1.0f : 0.0f) : v) - P.mf;
                        atomicOr(&sh.mask[s], 1 << c);
                    }
                    sh.slot[c][lane + 32 * e] = (unsigned char)s;
                }
        };
        if constexpr (RPL == 1)
        {
            for (int c0 = 0; c0 < w; c0 += 4)
            {
                int2 rec[4][RPL];
#pragma unroll
                for (int u = 0; u < 4; ++u) load(c0 + u, rec[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u) insert(c0 + u, rec[u]);
            }
        }
        else
        {
            // one copy of the code, the loads three cells ahead: with up to 64 neighbours
            // the kernel's eight warps wait for its instructions more than for anything
            // else (9.5M systems of clustered data: 58.7 -> 54.5 ms; with up to 32 the
            // four copies above are 2 to 10 % faster)
            int2 rec[3][RPL];
#pragma unroll
            for (int u = 0; u < 3; ++u) load(u, rec[u]);
#pragma unroll 1
            for (int c = 0; c < w; ++c)
            {
                insert(c, rec[0]);
#pragma unroll
                for (int e = 0; e < RPL; ++e)
                {
                    rec[0][e] = rec[1][e];
                    rec[1][e] = rec[2][e];
                }
                load(c + 3, rec[2]);
            }
        }
        over = __any_sync(FULL, over);
        __syncwarp();

        // ---- the group: the largest of w, w/2, .. first cells that can share
        int gn = over ? 1 : w;
        int cb = 0, ur = 0;
        int my_ne = 0; // lane c: extras of cell c
        const int n0 = __shfl_sync(FULL, my.y, 0);
        for (; gn >= 2; gn = (gn + 1) / 2)
        {
            const unsigned gm = (1u << gn) - 1u;
            cb = (__reduce_max_sync(FULL, lane < gn ? my.y : 0) + 7) / 8 - 1;
            // common neighbours in the first cell's order, 8 cb of them shared
            int nc = 0;
            unsigned shared = 0;
#pragma unroll
            for (int e = 0; e < RPL; ++e)
            {
                const int i = lane + 32 * e;
                const int sl = i < n0 ? sh.slot[0][i] : 0;
                const bool com = i < n0 && ((unsigned)sh.mask[sl] & gm) == gm;
                const unsigned b = __ballot_sync(FULL, com);
                const int rank = nc + __popc(b & below);
                if (com && rank < 8 * cb)
                {
                    const int at = HALVES ? mma_slot(rank, 8 * cb, cb) : rank;
                    sh.clin[at] = sh.key[sl];
                    sh.cval[at] = sh.val[sl];
                    sh.id[sl] = 255;
                    shared |= 1u << e;
                }
                nc += __popc(b);
            }
            if (cb < 1 || nc < 8 * cb)
            {
                __syncwarp(); // the next size writes clin, cval and id from other lanes
                continue;
            }
            // the distinct extras, each numbered by its first cell, and the
            // extras of every cell as rows of R
            ur = 0;
            for (int c = 0; c < gn; ++c)
            {
                const int n = __shfl_sync(FULL, my.y, c);
                int sl[RPL];
#pragma unroll
                for (int e = 0; e < RPL; ++e)
                {
                    const int i = lane + 32 * e;
                    sl[e] = i < n ? sh.slot[c][i] : -1;
                    const unsigned m = sl[e] >= 0 ? (unsigned)sh.mask[sl[e]] & gm : 0u;
                    const bool own = __ffs(m) - 1 == c && !(c == 0 && (shared >> e & 1));
                    const unsigned b = __ballot_sync(FULL, own);
                    const int id = min(ur + __popc(b & below), 254);
                    if (own)
                    {
                        sh.id[sl[e]] = (unsigned char)id;
                        if (id < kShareRows)
                        {
                            sh.rlin[id] = sh.key[sl[e]];
                            sh.rval[id] = sh.val[sl[e]];
                        }
                    }
                    ur += __popc(b);
                }
                __syncwarp();
                int ne = 0;
#pragma unroll
                for (int e = 0; e < RPL; ++e)
                {
                    const int id = sl[e] >= 0 ? sh.id[sl[e]] : 255;
                    const unsigned b = __ballot_sync(FULL, id != 255);
                    if (id != 255) sh.eid[c][ne + __popc(b & below)] = (unsigned char)id;
                    ne += __popc(b);
                }
                if (lane == c) my_ne = ne;
            }
            if (ur + gn + Q - 1 <= kShareRows) break;
            __syncwarp();
        }
        if (gn < 2)
        {
            // nothing shared: the one-system-per-warp kernel
            if (lane == 0) left_cells[atomicAdd(left_count, 1)] = my;
            __syncwarp();
            base += 1;
            continue;
        }
        if (lane < gn) sh.rlin[ur + lane] = my_off;
        __syncwarp();
        {
            // ---- the common block, factored once
            Blk A[1][CB * (CB + 1) / 2], none[1];
            bool fail[1] = {false};
            mma_load<CB>(A[0], pair_c, sh.clin, 8 * cb, cb, lane);
            if constexpr (HALVES)
                half_factor<CB, false, false, true>(A[0], none, cb, sh.row, lane, fail[0]);
            else
                mma_factor<CB, 1>(A, cb, sh.row, lane, fail);

            // ---- the rows of R, eight at a time
            const int rows = ur + gn + Q - 1;
            for (int rb = 0; rb < rows; rb += 8)
            {
                const int rho = rb + r;
                const bool gather = rho < ur + gn;
                const int rl = gather ? sh.rlin[rho] : 0;
                Blk R[CB];
#pragma unroll
                for (int k = 0; k < CB; ++k)
                {
                    if (k >= cb) break;
                    const int col = 8 * k + 2 * q;
                    const int2 lc = *reinterpret_cast<const int2 *>(&sh.clin[col]);
                    R[k] = Blk{0.0, 0.0};
                    if (gather)
                    {
                        R[k].x = __ldg(pair_c + abs(rl - lc.x));
                        R[k].y = __ldg(pair_c + abs(rl - lc.y));
                    }
                    else if (rho == rows - 1)
                    {
                        R[k].x = (double)sh.cval[col];
                        R[k].y = (double)sh.cval[col + 1];
                    }
                    else if (rho < rows)
                        R[k].x = R[k].y = 1.0;
                }
#pragma unroll
                for (int k = 0; k < CB; ++k)
                {
                    if (k >= cb) break;
                    const Blk &D = A[0][blk_at(k, k)];
                    Blk t = HALVES ? blk_solve_t(R[k], D) : blk_prod_t(R[k], D);
                    reinterpret_cast<double2 *>(&sh.R[rho * LD + 8 * k])[q] = make_double2(t.x, t.y);
                    t = blk_neg(t);
#pragma unroll
                    for (int j = k + 1; j < CB; ++j)
                    {
                        if (j >= cb) break;
                        blk_mul_t(R[j], t, A[0][blk_at(j, k)]);
                    }
                }
            }
            __syncwarp();

            // ---- the common part of the forms: four lanes per cell
            {
                double f[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
                const double2 *Rb = reinterpret_cast<const double2 *>(&sh.R[(ur + min(r, gn - 1)) * LD]);
                const double2 *R1 = reinterpret_cast<const double2 *>(&sh.R[(rows - 2) * LD]);
                const double2 *Rv = reinterpret_cast<const double2 *>(&sh.R[(rows - 1) * LD]);
#pragma unroll
                for (int k = 0; k < CB; ++k)
                {
                    if (k >= cb) break;
                    const double2 b = Rb[4 * k + q], v = Rv[4 * k + q];
                    f[0] = fma(b.x, b.x, fma(b.y, b.y, f[0]));
                    f[Q - 1] = fma(b.x, v.x, fma(b.y, v.y, f[Q - 1]));
                    if (ORDINARY)
                    {
                        const double2 o = R1[4 * k + q];
                        f[1] = fma(b.x, o.x, fma(b.y, o.y, f[1]));
                        f[3] = fma(o.x, o.x, fma(o.y, o.y, f[3]));
                        f[4] = fma(o.x, v.x, fma(o.y, v.y, f[4]));
                    }
                }
#pragma unroll
                for (int i = 0; i < 5; ++i)
                {
                    if (!ORDINARY && i >= 2) break;
                    f[i] += __shfl_xor_sync(FULL, f[i], 1);
                    f[i] += __shfl_xor_sync(FULL, f[i], 2);
                    if (q == 0) sh.F[r][i] = f[i];
                }
            }

            // ---- each cell's Schur complement, then its elimination, four cells a time
            bool bad = fail[0];
            for (int c4 = 0; c4 < gn; c4 += 4)
            {
                const int nu = min(4, gn - c4);
                int nemax = 0;
                for (int u = 0; u < nu; ++u)
                {
                    const int c = c4 + u;
                    const int ne = __shfl_sync(FULL, my_ne, c);
                    const int off = __shfl_sync(FULL, my_off, c);
                    nemax = max(nemax, ne);
                    const bool lr = r < ne, l0 = 2 * q < ne, l1 = 2 * q + 1 < ne;
                    const int er = lr ? sh.eid[c][r] : 0;
                    const int e0 = l0 ? sh.eid[c][2 * q] : 0, e1 = l1 ? sh.eid[c][2 * q + 1] : 0;
                    const int lr_lin = sh.rlin[er], l0_lin = sh.rlin[e0], l1_lin = sh.rlin[e1];
                    Blk S, X{0.0, 0.0};
                    S.x = lr && l0 ? __ldg(pair_c + abs(lr_lin - l0_lin)) : (r == 2 * q ? 1.0 : 0.0);
                    S.y = lr && l1 ? __ldg(pair_c + abs(lr_lin - l1_lin)) : (r == 2 * q + 1 ? 1.0 : 0.0);
                    if (r == 0)
                    {
                        X.x = l0 ? __ldg(pair_c + abs(l0_lin - off)) : 0.0;
                        X.y = l1 ? __ldg(pair_c + abs(l1_lin - off)) : 0.0;
                    }
                    else if (r == Q - 1)
                    {
                        X.x = l0 ? (double)sh.rval[e0] : 0.0;
                        X.y = l1 ? (double)sh.rval[e1] : 0.0;
                    }
                    else if (r < Q)
                    {
                        X.x = l0 ? 1.0 : 0.0;
                        X.y = l1 ? 1.0 : 0.0;
                    }
                    // row of the right-hand sides in R: b of the cell, ones, values
                    const int xr = r == 0 ? ur + c : rows - Q + r;
#pragma unroll
                    for (int k = 0; k < CB; ++k)
                    {
                        if (k >= cb) break;
                        double2 e = make_double2(0.0, 0.0), x = make_double2(0.0, 0.0);
                        if (lr) e = reinterpret_cast<const double2 *>(&sh.R[er * LD + 8 * k])[q];
                        if (r < Q) x = reinterpret_cast<const double2 *>(&sh.R[xr * LD + 8 * k])[q];
                        const Blk E{e.x, e.y};
                        const Blk En = blk_neg(E);
                        blk_mul_t(S, En, E);
                        blk_mul_t(X, Blk{x.x, x.y}, En);
                    }
                    reinterpret_cast<double2 *>(sh.S[u])[4 * r + (q ^ ((r >> 1) & 3))] = make_double2(S.x, S.y);
                    if (r < Q) reinterpret_cast<double2 *>(sh.XE[u])[4 * r + q] = make_double2(X.x, X.y);
                }
                __syncwarp();
                // lane 8 u + t: row t of cell u's system
                const int u = min(lane >> 3, nu - 1), t = lane & 7;
                double a[8], z[Q];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                {
                    const double2 v = reinterpret_cast<const double2 *>(sh.S[u])[4 * t + (i ^ ((t >> 1) & 3))];
                    a[2 * i] = v.x;
                    a[2 * i + 1] = v.y;
                }
#pragma unroll
                for (int i = 0; i < Q; ++i) z[i] = sh.XE[u][8 * i + t];
                // form of the lane: (0,0) (0,1) (0,2) (1,1) (1,2)
                const int ia = t >= 3 ? 1 : 0, ib = t >= 3 ? t - 2 : t;
                const bool form = t < (ORDINARY ? 5 : 2);
                double acc = 0.0;
                bool bad_u = false;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                {
                    if (j >= nemax) break;
                    double *buf = sh.row + (j & 1) * 48 + (lane >> 3) * 12;
                    if (t == j)
                    {
#pragma unroll
                        for (int i = j / 2; i < 4; ++i)
                            reinterpret_cast<double2 *>(buf)[i] = make_double2(a[2 * i], a[2 * i + 1]);
#pragma unroll
                        for (int i = 0; i < Q; ++i) buf[8 + i] = z[i];
                    }
                    __syncwarp();
                    const double p = buf[j];
                    bad_u |= pivot_fails<false>(p);
                    const double inv = pivot_inverse(p);
                    const double m = t > j ? a[j] * inv : 0.0;
#pragma unroll
                    for (int i = (j + 1) / 2; i < 4; ++i)
                    {
                        const double2 v = reinterpret_cast<const double2 *>(buf)[i];
                        if (2 * i > j) a[2 * i] = fma(-m, v.x, a[2 * i]);
                        a[2 * i + 1] = fma(-m, v.y, a[2 * i + 1]);
                    }
#pragma unroll
                    for (int i = 0; i < Q; ++i) z[i] = fma(-m, buf[8 + i], z[i]);
                    if (form) acc = fma(buf[8 + ia] * inv, buf[8 + ib], acc);
                }
                if (lane < 8 * nu && form) sh.F[c4 + (lane >> 3)][t] += acc;
                if (lane < 8 * nu && t == 7) sh.F[c4 + (lane >> 3)][5] = bad_u ? 1.0 : 0.0;
                __syncwarp();
            }
            // ---- forms -> estimates: lane c writes cell c
            if (lane < gn)
            {
                const double *f = sh.F[lane];
                if (bad || f[5] != 0.0)
                    left_cells[atomicAdd(left_count, 1)] = my;
                else
                    write_solution<ORDINARY>(P, my.x, false, f[Q - 1], f[0], f[1], f[4], f[3]);
            }
            __syncwarp();
        }
        base += gn;
    }
}

template <int CB, bool ORD, int TH, bool HALVES>
static cudaError_t launch_share(const Geom &g, const int2 *cells, const int *n_items, int max_items, const int2 *nb_rec,
                                int ind_value, const SolveParams &P, const CellTile &tile, int2 *left_cells, int *left_count,
                                int n_sm, cudaStream_t st)
{
    const size_t smem = sizeof(ShareWarp<CB>) * (TH / 32);
    auto kern = k_solve_share<CB, ORD, TH, HALVES>;
    int blocks = 0;
    cudaError_t e = launch_kernel(kern, TH, smem, max_items, TH / 32 * kShareCells, n_sm, blocks);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)blocks, TH, smem, st>>>(g, cells, n_items, nb_rec, ind_value, P, tile, left_cells, left_count);
    return cudaGetLastError();
}

// The tile whose cells a group is taken from: eight cells as 2^lx x 2^ly x 2^lz,
// the shape with the least summed displacement relative to the search radiuses
// (a displaced neighbourhood loses points in proportion). Limits per axis: the
// grid's own extent, and the offsets of any two neighbours of two of its cells
// must still tell the points apart (|dx| below the table's row length, |dy|
// below its row count).
CellTile solve_share_tile(const Geom &g)
{
    // the neighbours' reach per axis: analytic tables, box-truncated ones
    const int hx = g.phx >= 4 * g.rx - 2 ? g.khx : g.rx, hy = g.phy >= 4 * g.ry - 2 ? g.khy : g.ry;
    const int mx = g.pnx - 2 * hx < g.nx ? g.pnx - 2 * hx : g.nx;
    const int my = g.pny - 2 * hy < g.ny ? g.pny - 2 * hy : g.ny;
    CellTile best{0, 0, 0};
    double cost = 0.0;
    int cells = 0;
    for (int lx = 0; lx <= 3; ++lx)
        for (int ly = 0; lx + ly <= 3; ++ly)
            for (int lz = 0; lx + ly + lz <= 3; ++lz)
            {
                if ((1 << lx) > mx || (1 << ly) > my || (1 << lz) > g.nz) continue;
                const double c = ((1 << lx) - 1) / (double)g.rx + ((1 << ly) - 1) / (double)g.ry +
                                 ((1 << lz) - 1) / (double)g.rz;
                const int n = 1 << (lx + ly + lz);
                if (n > cells || (n == cells && c < cost))
                {
                    best = CellTile{lx, ly, lz};
                    cost = c;
                    cells = n;
                }
            }
    return best;
}

cudaError_t launch_solve_share(int np, bool ordinary, const Geom &g, const int2 *cells, const int *n_items,
                               int max_items, const int2 *nb_rec, int ind_value, const SolveParams &P, const CellTile &tile,
                               int2 *left_cells, int *left_count, int n_sm, cudaStream_t st)
{
#define HB_ARGS g, cells, n_items, max_items, nb_rec, ind_value, P, tile, left_cells, left_count, n_sm, st
#define HB_SHARE(CB, TH)                                                                         \
    (P.out.by_halves ? (ordinary ? launch_share<CB, true, TH, true>(HB_ARGS) : launch_share<CB, false, TH, true>(HB_ARGS)) \
              : (ordinary ? launch_share<CB, true, TH, false>(HB_ARGS) : launch_share<CB, false, TH, false>(HB_ARGS)))
    if (np == 32) return HB_SHARE(3, 512);
    if (np == 64) return HB_SHARE(7, 256);
    return cudaErrorInvalidValue;
#undef HB_SHARE
#undef HB_ARGS
}
} // namespace hb
