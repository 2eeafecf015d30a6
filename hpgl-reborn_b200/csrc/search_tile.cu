// Neighbour selection, one cell a lane (the reference's lookups; see search.cu for
// the warp-per-cell forms).
#include "engine.cuh"
#include "kernels.h"
#include "search_common.cuh"

#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

namespace hb
{
// One cell by exact ranks over all C candidates, without scratch: the smallest
// rank with k candidates up to it by bisection, then those candidates' keys (rank
// << 16 | place) to out, ld apart. Returns the neighbour count, or -1 for a tie
// group across the k-th slot.
__device__ int exact_select(const Geom &g, int C, const float4 *ctp, int kofs, const uint16_t *__restrict__ keytab,
                            int lane, uint32_t *out, int ld)
{
    const int k = g.k;
    auto rank = [&](int i) { return (int)keytab[kofs + __float_as_int(ctp[i].w)]; };
    auto count = [&](int top) {
        int c = 0;
        for (int i = lane; i < C; i += 32) c += rank(i) <= top;
        return __reduce_add_sync(0xffffffffu, c);
    };
    int lo = -1, hi = 0xFFFE; // kept ranks stay below 0xFFFF
    const int kept = count(hi);
    int at = kept;
    if (kept > k)
        while (at != k)
        {
            if (hi - lo == 1) return -1;
            const int mid = (lo + hi) >> 1;
            const int c = count(mid);
            if (c >= k)
            {
                hi = mid;
                at = c;
            }
            else
                lo = mid;
        }
    int done = 0;
    for (int base = 0; base < C; base += 32)
    {
        const int i = base + lane, r = i < C ? rank(i) : 0xFFFF;
        const unsigned bl = __ballot_sync(0xffffffffu, r <= hi);
        if (r <= hi) out[(done + __popc(bl & lanemask_lt())) * ld] = ((uint32_t)r << 16) | (uint32_t)i;
        done += __popc(bl);
    }
    return done;
}

// ---- ascending order of a lane's own keys: Batcher's odd-even merge sort (K. E.
// Batcher, Sorting networks and their applications, 1968) on registers. A lane has
// its list to itself, so 32 cells' lists of 32 take 191 comparators, about 14 warp
// instructions a cell; sorted across the warp a cell at a time, 60.
template <int A, int B, int N>
__device__ __forceinline__ void compare_exchange(uint32_t (&v)[N])
{
    const uint32_t lo = min(v[A], v[B]);
    v[B] = max(v[A], v[B]);
    v[A] = lo;
}
template <int FIRST, int LEN, int STEP, int I, int N>
__device__ __forceinline__ void merge_pairs(uint32_t (&v)[N])
{
    if constexpr (I + STEP < FIRST + LEN)
    {
        compare_exchange<I, I + STEP>(v);
        merge_pairs<FIRST, LEN, STEP, I + 2 * STEP>(v);
    }
}
template <int FIRST, int LEN, int STEP, int N>
__device__ __forceinline__ void odd_even_merge(uint32_t (&v)[N])
{
    if constexpr (2 * STEP < LEN)
    {
        odd_even_merge<FIRST, LEN, 2 * STEP>(v);
        odd_even_merge<FIRST + STEP, LEN, 2 * STEP>(v);
        merge_pairs<FIRST, LEN, STEP, FIRST + STEP>(v);
    }
    else
        compare_exchange<FIRST, FIRST + STEP>(v);
}
template <int FIRST, int LEN, int N>
__device__ __forceinline__ void merge_sort(uint32_t (&v)[N])
{
    if constexpr (LEN > 1)
    {
        merge_sort<FIRST, LEN / 2>(v);
        merge_sort<FIRST + LEN / 2, LEN / 2>(v);
        odd_even_merge<FIRST, LEN, 1>(v);
    }
}

constexpr uint32_t kNoKey = 0xFFFFFFFFu; // past every key

// the N keys from `first` on of a lane's list of n, ld apart
template <int N, int P>
__device__ __forceinline__ void load_keys(uint32_t (&v)[P], const uint32_t *list, int ld, int first, int n)
{
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] = first + e < n ? list[(first + e) * ld] : kNoKey;
}
template <int N, int P>
__device__ __forceinline__ void store_keys(const uint32_t (&v)[P], uint32_t *list, int ld, int first, int n)
{
#pragma unroll
    for (int e = 0; e < N; ++e)
        if (first + e < n) list[(first + e) * ld] = v[e];
}
// (a function of its own: inlined, its registers drove the search's to local memory,
// 4.3 -> 7.3 ms; 4.75 so)
template <int N>
__device__ __noinline__ void order_keys(uint32_t *list, int ld, int first, int n)
{
    constexpr int P = N <= 8 ? 8 : (N <= 16 ? 16 : 32);
    uint32_t v[P];
    load_keys<N>(v, list, ld, first, n);
#pragma unroll
    for (int e = N; e < P; ++e) v[e] = kNoKey; // the compiler drops their comparators
    merge_sort<0, P>(v);
    store_keys<N>(v, list, ld, first, n);
}
// a bitonic run of 32 put in order
__device__ __forceinline__ void order_bitonic(uint32_t (&v)[32])
{
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (!(i & s))
            {
                const uint32_t lo = min(v[i], v[i + s]);
                v[i + s] = max(v[i], v[i + s]);
                v[i] = lo;
            }
}
// 33 to 64 keys: two sorted halves, the i-th of the first against the (31 - i)-th of
// the second, then two bitonic runs (64 registers would not fit beside the search's)
__device__ __noinline__ void order_keys64(uint32_t *list, int ld, int n)
{
#pragma unroll 1
    for (int h = 0; h < 64; h += 32) order_keys<32>(list, ld, h, n);
    uint32_t v[32];
    load_keys<32>(v, list, ld, 0, n);
#pragma unroll
    for (int i = 0; i < 32; ++i)
    {
        const int at = 63 - i;
        if (at < n)
        {
            const uint32_t x = list[at * ld];
            list[at * ld] = max(v[i], x);
            v[i] = min(v[i], x);
        }
    }
    order_bitonic(v);
    store_keys<32>(v, list, ld, 0, n);
    // the upper half: bitonic with kNoKey from n on
    load_keys<32>(v, list, ld, 32, n);
    order_bitonic(v);
    store_keys<32>(v, list, ld, 32, n);
}

// ---- the same selection, one cell a lane
//
// A warp takes a tile of 32 cells of a bin (a few cells in each direction, so
// that their neighbourhoods nearly coincide) and lists the candidates near the
// tile once; each lane then scans that list for its own cell, keeps the
// candidates inside its radius, reads their exact ranks, finds the k-th by
// counting, and decides as select_surr does, with the same bounds. A cell's work
// is about a tenth of the warp-per-cell form's (whose every step costs a warp
// instruction for one cell). Lanes whose radius was a bad guess repeat the scan
// with another; what is undecided after kTileTries goes through exact_select.
// Neighbours are written in key order, equal ranks in candidate order: the nearest
// first is also what keeps the solves' rounding low (12 neighbours, Gaussian, nugget
// 0.05, simple kriging: in candidate order 2.2 times the estimates' error and 1.5 times
// the variances'). The sort of each lane's list costs 0.5 of 4.8 ms at 8.3M cells of 32,
// 2 of 48 ms at 16.8M clustered cells of 64, 0.8 of 13.2 ms at 20M indicator cells of 24.
//
// What bounds it: instructions (on a grid of 32 neighbours about half the issue
// slots, on clustered data of 64 a third, where the lists leave room for 14 warps
// on an SM). So every loop runs to the warp's longest list, in fours: a lane that
// stopped at its own list's end cost the others a pass more, and loads between
// stores to the list waited one after another. The rank search ends by ordering the
// last kTileFinal survivors, since one lane with a tie in 32 would take every lane
// through a full bisection (6 in place of 4: 4.5 against 4.3 ms). Measured, with
// each lane to its own end and bisection alone before: 8.3M cells of 32 neighbours
// 4.73 -> 4.28 ms, 16.8M clustered cells of 64 58.9 -> 45.7 ms, 20M indicator cells
// 14.3 -> 12.4 ms. Blocks of up to 12 warps gain 2 % on clustered data and lose
// 14 % on 500,000 sparse cells.
constexpr int kTileTries = 8;
constexpr int kTileFinal = 4; // survivors that the rank search puts in order at its end
constexpr int kManyCandidates = 1024; // candidates of a bin away from data clusters

struct SearchTile
{
    int ty, tz;  // rows and layers of a tile (32 / (ty tz) cells along x)
    int cap;     // survivors a lane keeps
    int sub;     // candidates near a tile, at most (beyond: all are scanned)
    int slices;  // blocks per bin
    int c_min, c_max; // the bins of this launch: c_min < candidates <= c_max
    bool leave_scans; // and not those that are better scanned
};

__global__ void __launch_bounds__(256, 3) k_search_tile(
    const Geom g, const uint8_t *__restrict__ mask, int all_cells, const int *__restrict__ bin_start,
    const int *__restrict__ bin_cnt, const uint8_t *__restrict__ bin_flag, const int *__restrict__ bin_pts,
    const unsigned long long *__restrict__ pts_xyz, const float *__restrict__ pts_vf,
    const uint16_t *__restrict__ keytab, const SurrDev sd, const SearchTile tl, int template_bins, int cand_cap,
    int2 *__restrict__ nb_rec, int *__restrict__ nb_n, int *__restrict__ tie_cells, int *__restrict__ tie_count,
    int *__restrict__ n_template_cells, int *__restrict__ exact_cells)
{
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char smem[];
    const int b = blockIdx.x / tl.slices, slice = blockIdx.x % tl.slices;
    const int bxi = b % g.bx, byi = (b / g.bx) % g.by, bzi = b / (g.bx * g.by);
    const int x0 = bxi * g.rx, y0 = byi * g.ry, z0 = bzi * g.rz;
    if (x0 >= g.nx || y0 >= g.ny || z0 >= g.nz) return;
    if (((bin_flag[b] >> 1) & 1) != template_bins) return;
    const int wx = min(g.rx, g.nx - x0), wy = min(g.ry, g.ny - y0), wz = min(g.rz, g.nz - z0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int k = g.k, cap = tl.cap, ld = blockDim.x + 1;

    float4 *ctp = reinterpret_cast<float4 *>(smem);
    int2 *crec = reinterpret_cast<int2 *>(ctp + cand_cap); // pair-table offset from the bin corner, value
    uint32_t *lists = reinterpret_cast<uint32_t *>(crec + cand_cap); // [cap][threads + 1]
    uint32_t *list = lists + threadIdx.x;
    uint16_t *sub = reinterpret_cast<uint16_t *>(lists + (size_t)cap * ld) + warp * tl.sub;

    // candidates of the 27 bins around, in the reference's order: every thread
    // finds its own in the nine runs, so that their dependent loads (point,
    // coordinates, value) are waited for together (a bin at a time, a block with
    // few candidates waited 27 times)
    __shared__ int s_pre[16], s_start[16], s_total;
    if (threadIdx.x < 32)
    {
        const int c = candidate_runs(g, bxi, byi, bzi, bin_start, bin_cnt, threadIdx.x, s_pre, s_start);
        if (threadIdx.x == 0) s_total = c;
    }
    __syncthreads();
    const int C = s_total;
    if (C <= tl.c_min || C > tl.c_max) return;
    if (tl.leave_scans && scan_is_shorter(g, bxi, byi, bzi, C, bin_cnt[b])) return;
#pragma unroll 2
    for (int d = threadIdx.x; d < C; d += blockDim.x)
    {
        const int q = run_of(s_pre, d);
        const int p = bin_pts[s_start[q] + d - s_pre[q]];
        int px, py, pz;
        unpack_xyz(pts_xyz[p], px, py, pz);
        // float coordinates, and the offset into the key table from the bin corner
        float4 c = surr_coords(sd, px - x0, py - y0, pz - z0);
        c.w = __int_as_float(((pz - z0) * g.kny + (py - y0)) * g.knx + (px - x0));
        ctp[d] = c;
        crec[d] = make_int2(pair_lin(g, px - x0, py - y0, pz - z0), __float_as_int(pts_vf[p]));
    }
    __syncthreads();
    const int kc0 = (g.khz * g.kny + g.khy) * g.knx + g.khx;
    const float e3 = (float)sd.e3 * (1.0f + 1e-6f) + 1e-30f;
    const float r_all = (float)(sd.h_cut * (1.0 + 1e-5) + 4.0 * sd.e3); // decides every candidate
    // radius that holds 1.25 k of C candidates spread over 27 bins
    float guess = cbrtf(1.25f * (float)k * 27.0f * (float)g.rx * (float)g.ry * (float)g.rz / (4.18879f * (float)max(C, 1)) *
                        sd.step[0] * sd.step[1] * sd.step[2]);

    const int ny_s = (wy + tl.ty - 1) / tl.ty, nz_s = (wz + tl.tz - 1) / tl.tz;
    const int parts = (wx * min(tl.ty, wy) * min(tl.tz, wz) + 31) / 32;
    const int n_tiles = ny_s * nz_s * parts;
    const int per = (n_tiles + tl.slices * nwarps - 1) / (tl.slices * nwarps);
    const int t0 = (slice * nwarps + warp) * per, t1 = min(t0 + per, n_tiles);
    int n_exact = 0, n_done = 0;
    for (int tile = t0; tile < t1; ++tile)
    {
        // ---- the lane's cell: rows and layers fastest, then x
        const int part = tile % parts, ys = tile / parts % ny_s, zs = tile / parts / ny_s;
        const int hy = min(tl.ty, wy - ys * tl.ty), hz = min(tl.tz, wz - zs * tl.tz);
        const int t = part * 32 + lane, col = hy * hz;
        const int cxr = min(t / col, wx - 1), cyr = ys * tl.ty + t % col % hy, czr = zs * tl.tz + t % col / hy;
        const long long cell = ((long long)(z0 + czr) * g.ny + (y0 + cyr)) * g.nx + (x0 + cxr);
        bool open = t < col * wx && (all_cells || !mask[cell]);
        if (!__any_sync(FULL, open)) continue;
        n_done += __popc(__ballot_sync(FULL, open));
        const float4 tc = surr_coords(sd, cxr, cyr, czr);
        const int klin_c = (czr * g.kny + cyr) * g.knx + cxr;
        // the tile's centre and the lane's distance from it
        float ccx, ccy, ccz, dc;
        {
            const float4 c0 = make_float4(__shfl_sync(FULL, tc.x, 0), __shfl_sync(FULL, tc.y, 0),
                                          __shfl_sync(FULL, tc.z, 0), 0.0f);
            const float4 c1 = make_float4(__shfl_sync(FULL, tc.x, 31), __shfl_sync(FULL, tc.y, 31),
                                          __shfl_sync(FULL, tc.z, 31), 0.0f);
            ccx = 0.5f * (c0.x + c1.x);
            ccy = 0.5f * (c0.y + c1.y);
            ccz = 0.5f * (c0.z + c1.z);
            const float dx = tc.x - ccx, dy = tc.y - ccy, dz = tc.z - ccz;
            dc = sqrtf(fmaf(dz, dz, fmaf(dy, dy, dx * dx)));
        }
        // the lane's radius: known to keep fewer than k at lo_r, more than cap at hi_r
        float rt = fminf(guess, r_all), lo_r = 0.0f, hi_r = 0.0f, H = 0.0f;
        float lo_c = 0.0f, hi_c = 0.0f, have = -1.0f; // have: reach of the list in `sub`
        int n = -2, n_sub = 0;
        bool all = false;
        for (int tries = 0; tries < kTileTries; ++tries)
        {
            // ---- candidates within reach of any open lane: every candidate whose float
            // distance from the centre exceeds R is truly farther than R - e3 - rounding
            // from it, so farther than rt + e3 from a lane's cell at dc + e3 from it
            float reach = open ? (rt + dc) * (1.0f + 1e-5f) + 4.0f * e3 : 0.0f;
            reach = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(reach)));
            if (reach > have)
            {
                have = reach;
                const float R2 = reach * reach * (1.0f + 1e-5f);
                n_sub = 0;
                __syncwarp();
                for (int base = 0; base < C; base += 32)
                {
                    const int i = base + lane;
                    bool in = false;
                    if (i < C)
                    {
                        const float4 c = ctp[i];
                        const float dx = c.x - ccx, dy = c.y - ccy, dz = c.z - ccz;
                        in = fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= R2;
                    }
                    const unsigned bl = __ballot_sync(FULL, in);
                    const int at = n_sub + __popc(bl & lanemask_lt());
                    if (in && at < tl.sub) sub[at] = (uint16_t)i;
                    n_sub += __popc(bl);
                }
                all = n_sub > tl.sub;
                if (all) n_sub = C;
                __syncwarp();
            }
            // ---- the lane's scan, four candidates' loads at a time (a store to the list
            // between them would keep the compiler from issuing the next load)
            const float Tg = __fmul_ru(__fmul_ru(rt, rt), 1.0f + 1e-6f);
            int cnt = open ? 0 : cap + 1;
            for (int j = 0; j < n_sub; j += 4)
            {
                int at[4];
                float4 c[4];
                const uint2 s4 = reinterpret_cast<const uint2 *>(sub)[all ? 0 : j >> 2];
                at[0] = all ? j : (int)(s4.x & 0xFFFFu);
                at[1] = all ? j + 1 : (int)(s4.x >> 16);
                at[2] = all ? j + 2 : (int)(s4.y & 0xFFFFu);
                at[3] = all ? j + 3 : (int)(s4.y >> 16);
#pragma unroll
                for (int u = 0; u < 4; ++u) c[u] = ctp[j + u < n_sub ? at[u] : 0];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                {
                    const float qx = c[u].x - tc.x, qy = c[u].y - tc.y, qz = c[u].z - tc.z;
                    if (fmaf(qz, qz, fmaf(qy, qy, qx * qx)) <= Tg && j + u < n_sub)
                    {
                        if (cnt < cap) list[cnt * ld] = (uint32_t)at[u];
                        ++cnt;
                    }
                }
            }
            // ---- the lane's decision
            const bool few = open && cnt < k && rt < r_all, many = open && cnt > cap;
            if (few)
            {
                lo_r = rt;
                lo_c = (float)cnt;
            }
            if (many)
            {
                hi_r = rt;
                hi_c = (float)cnt;
            }
            if (few || many)
            {
                // between both bounds by their counts, else by the volume
                const float goal = 0.5f * (float)(k + cap);
                if (lo_r > 0.0f && hi_r > 0.0f)
                    rt = lo_r + (hi_r - lo_r) * fminf(fmaxf((goal - lo_c) / (hi_c - lo_c), 0.1f), 0.9f);
                else if (few)
                    rt = fminf(rt * fminf(cbrtf(goal / fmaxf((float)cnt, 0.25f)) + 0.01f, 2.0f) + e3, r_all);
                else
                    rt = rt * fmaxf(cbrtf(goal / (float)cnt), 0.7f);
            }
            const bool ranked = open && !few && !many;
            // the loops over the lists run to the longest list of the warp, in fours:
            // no lane branches away from the others
            const int rows = (__reduce_max_sync(FULL, ranked ? cnt : 0) + 3) & ~3;
            if (ranked)
            {
                int nk = 0, rmin = 0x10000, rmax = -1;
                for (int e = 0; e < rows; e += 4)
                {
                    uint32_t pos[4];
                    int r16[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) pos[u] = e + u < cnt ? list[(e + u) * ld] : 0u;
#pragma unroll
                    for (int u = 0; u < 4; ++u) r16[u] = __float_as_int(ctp[pos[u]].w);
#pragma unroll
                    for (int u = 0; u < 4; ++u) r16[u] = keytab[kc0 - klin_c + r16[u]];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (r16[u] != 0xFFFF && e + u < cnt)
                        {
                            list[nk * ld] = ((uint32_t)r16[u] << 16) | pos[u];
                            ++nk;
                            rmin = min(rmin, r16[u]);
                            rmax = max(rmax, r16[u]);
                        }
                }
                for (int e = nk; e < rows; ++e) list[e * ld] = 0xFFFFFFFFu; // past every rank
                if (nk < k && rt < r_all)
                {
                    rt = r_all; // survivors without a rank: the kept offsets end near here
                }
                else
                {
                    // smallest rank T with k survivors up to it; a rank that holds the k-th
                    // and the (k+1)-th is a tie across the last slot. By interpolating counts
                    // (clo below k up to lo, chi above k up to hi) down to kTileFinal
                    // survivors between, which one pass then puts in order
                    int T = rmax;
                    bool tie = false;
                    if (nk > k)
                    {
                        int lo = rmin - 1, hi = rmax, clo = 0, chi = nk;
                        bool found = false;
                        for (int it = 0; chi - clo > kTileFinal && !found; ++it)
                        {
                            if (hi - lo == 1)
                            {
                                T = hi;
                                tie = found = true;
                                break;
                            }
                            int mid = (it & 3) == 3 ? (lo + hi) >> 1
                                                  : lo + (int)((float)(hi - lo) * ((float)(k - clo) + 0.5f) /
                                                               ((float)(chi - clo) + 0.5f));
                            mid = min(max(mid, lo + 1), hi - 1);
                            const uint32_t top = ((uint32_t)mid << 16) | 0xFFFFu;
                            int c = 0;
                            for (int e = 0; e < rows; e += 4)
#pragma unroll
                                for (int u = 0; u < 4; ++u) c += list[(e + u) * ld] <= top;
                            if (c == k)
                            {
                                T = mid;
                                found = true;
                            }
                            else if (c < k)
                            {
                                lo = mid;
                                clo = c;
                            }
                            else
                            {
                                hi = mid;
                                chi = c;
                            }
                        }
                        if (!found)
                        {
                            // the smallest kTileFinal survivors above lo; of them the
                            // (k - clo)-th and the next are there
                            const uint32_t bot = lo < 0 ? 0u : ((uint32_t)lo << 16) | 0xFFFFu;
                            uint32_t s[kTileFinal];
#pragma unroll
                            for (int i = 0; i < kTileFinal; ++i) s[i] = 0xFFFFFFFFu;
                            for (int e = 0; e < rows; e += 4)
#pragma unroll
                                for (int u = 0; u < 4; ++u)
                                {
                                    uint32_t x = list[(e + u) * ld];
                                    x = lo < 0 || x > bot ? x : 0xFFFFFFFFu;
#pragma unroll
                                    for (int i = 0; i < kTileFinal; ++i)
                                    {
                                        const uint32_t m = min(s[i], x);
                                        x = max(s[i], x);
                                        s[i] = m;
                                    }
                                }
                            uint32_t kth = s[0], next = s[1];
#pragma unroll
                            for (int i = 1; i < kTileFinal - 1; ++i)
                                if (k - clo > i)
                                {
                                    kth = s[i];
                                    next = s[i + 1];
                                }
                            T = (int)(kth >> 16);
                            tie = (kth >> 16) == (next >> 16);
                        }
                        // in place, the survivors up to T
                        const uint32_t top = ((uint32_t)T << 16) | 0xFFFFu;
                        int w = 0, last = 0;
                        for (int e = 0; e < rows; e += 4)
                        {
                            uint32_t key[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) key[u] = list[(e + u) * ld];
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                                if (key[u] <= top)
                                {
                                    last = max(last, (int)(key[u] >> 16));
                                    list[w * ld] = key[u];
                                    ++w;
                                }
                        }
                        T = last;
                    }
                    H = __double2float_ru(nk >= k ? sd.h_rank[T] : sd.h_cut);
                    if ((rt - e3) * (1.0f - 1e-6f) > H)
                    {
                        n = tie ? -1 : min(nk, k);
                        open = false;
                    }
                    else
                        rt = fminf(H * (1.0f + 4e-6f) + 3.0f * e3, r_all);
                }
            }
            if (!__any_sync(FULL, open)) break;
        }
        const bool mine = t < col * wx && (n != -2 || open);
        // ---- the next tile's radius: the largest k-th distance of this one
        {
            const float h = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(n != -2 ? H : 0.0f)));
            if (h > 0.0f) guess = h * 1.02f + e3;
        }
        // ---- undecided cells: by exact ranks over every candidate
        __syncwarp();
        for (unsigned todo = __ballot_sync(FULL, open); todo; todo &= todo - 1)
        {
            const int src = __ffs(todo) - 1;
            const int r = exact_select(g, C, ctp, kc0 - __shfl_sync(FULL, klin_c, src), keytab, lane,
                                       lists + warp * 32 + src, ld);
            if (lane == src) n = r;
            ++n_exact;
        }
        __syncwarp();
        // ---- the lists in key order
        const int own = mine ? max(n, 0) : 0, longest = __reduce_max_sync(FULL, own);
        if (longest > 32)
            order_keys64(list, ld, own);
        else if (longest > 24)
            order_keys<32>(list, ld, 0, own);
        else if (longest > 16)
            order_keys<24>(list, ld, 0, own);
        else if (longest > 8)
            order_keys<16>(list, ld, 0, own);
        else if (longest > 1)
            order_keys<8>(list, ld, 0, own);
        // ---- written a cell at a time
        __syncwarp();
        for (unsigned todo = __ballot_sync(FULL, own > 0); todo; todo &= todo - 1)
        {
            const int src = __ffs(todo) - 1;
            const int ns = __shfl_sync(FULL, n, src);
            const long long cs = __shfl_sync(FULL, cell, src);
            const int pl = __shfl_sync(FULL, pair_lin(g, cxr, cyr, czr), src);
            for (int e = lane; e < ns; e += 32)
            {
                const int2 rec = crec[lists[e * ld + warp * 32 + src] & 0xFFFFu];
                nb_rec[cs * k + e] = make_int2(rec.x - pl, rec.y);
            }
        }
        __syncwarp();
        if (mine)
        {
            nb_n[cell] = n < 0 ? k : n;
            if (n < 0) tie_cells[atomicAdd(tie_count, 1)] = (int)cell;
        }
    }
    if (exact_cells && lane == 0 && n_exact) atomicAdd(exact_cells, n_exact);
    if (template_bins && n_template_cells && lane == 0 && n_done) atomicAdd(n_template_cells, n_done);
}

// survivors a lane keeps, for k neighbours
static int tile_cap(int k) { return (k + std::max(12, k * 3 / 8 + 4) + 3) & ~3; } // in fours
static size_t tile_smem(int cand_cap, int cap, int sub, int warps)
{
    return (size_t)cand_cap * 24 + (size_t)cap * (warps * 32 + 1) * 4 + (size_t)warps * sub * 2;
}

// Shape of k_search_tile for a search: of the tiles with the most cells inside a bin of
// the grid (32, but for thin grids: taken by extent alone, the tile of a grid one
// cell wide was one cell, 2.4 in place of 0.46 ms for 200,000 of them), the one with
// the least extent in transformed coordinates; room for three eighths more survivors than
// neighbours, and the block size for the most warps on an SM; warps 0 when the candidates
// leave no room.
static SearchTile search_tile_shape(const Geom &g, const SurrDev &sd, int n_bins, int cand_cap, int max_smem, int &warps,
                                    size_t &smem)
{
    SearchTile t{1, 1, tile_cap(g.k), cand_cap <= kManyCandidates ? 256 : 1024, 1, 0, cand_cap, false};
    const int bx = std::min(g.rx, g.nx), by = std::min(g.ry, g.ny), bz = std::min(g.rz, g.nz);
    float best = 3.4e38f;
    int cells = 0;
    for (int ty = 1; ty <= 32; ty *= 2)
        for (int tz = 1; ty * tz <= 32; tz *= 2)
        {
            if ((ty > 1 && ty > by) || (tz > 1 && tz > bz)) continue;
            const int tx = std::min(32 / (ty * tz), bx), n = tx * ty * tz;
            const float ex = sd.step[0] * (float)tx, ey = sd.step[1] * ty, ez = sd.step[2] * tz;
            const float e = ex * ex + ey * ey + ez * ez;
            if (n > cells || (n == cells && e < best))
            {
                cells = n;
                best = e;
                t.ty = ty;
                t.tz = tz;
            }
        }
    const long long tiles = ((long long)g.rx * g.ry * g.rz + 31) / 32;
    // bins with many candidates leave room for few warps a block, and there may be few
    // bins: more blocks each, down to eight tiles a block
    const long long fill = (3552 + n_bins - 1) / n_bins;
    t.slices = (int)std::max<long long>(
        1, std::min(tiles / 8, std::max(tiles / (cand_cap > kManyCandidates ? 16 : 128), fill)));
    // the block size that keeps most warps on an SM (24 at most: 80 registers a thread)
    int most = 0;
    warps = 0;
    for (int w = 8; w > 0; --w)
    {
        const size_t need = tile_smem(cand_cap, t.cap, t.sub, w);
        if (need > (size_t)max_smem) continue;
        const int resident = std::min(24 / w, (int)(228 * 1024 / (need + 1024))) * w;
        if (resident > most)
        {
            most = resident;
            warps = w;
            smem = need;
        }
    }
    return t;
}

// Candidates of a bin that leave room for `warps` warps a block, at k neighbours.
int search_tile_limit(int k, int max_smem, int warps)
{
    const long long room = (long long)max_smem - (long long)tile_smem(0, tile_cap(k), 1024, warps);
    return (int)std::max(0LL, std::min(room / 24 / 4 * 4, 65536LL));
}

cudaError_t launch_search_tile(const Geom &g, const uint8_t *mask, int all_cells, const int *bin_start,
                               const int *bin_cnt, const uint8_t *bin_flag, const int *bin_pts,
                               const unsigned long long *pts_xyz, const float *pts_vf, const uint16_t *keytab16,
                               const SurrDev &sd, int template_bins, int n_bins, int cand_cap, int limit, bool leave_scans,
                               int max_smem, int2 *nb_rec,
                               int *nb_n, int *tie_cells, int *tie_count, int *n_template_cells, int *exact_cells,
                               cudaStream_t st)
{
    cand_cap = std::min(cand_cap, limit);
    if (cand_cap <= 0) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k_search_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
    if (e != cudaSuccess) return e;
    // the bins around data clusters in launches of their own: their candidates would
    // take the shared memory of every other bin's block too
    for (int c_min = -1, c_max = std::min(cand_cap, kManyCandidates);;)
    {
        int warps = 0;
        size_t smem = 0;
        SearchTile tl = search_tile_shape(g, sd, n_bins, c_max, max_smem, warps, smem);
        if (warps <= 0) return cudaErrorInvalidValue;
        tl.c_min = c_min;
        tl.c_max = c_max;
        tl.leave_scans = leave_scans;
        k_search_tile<<<(unsigned)((long long)g.n_bins * tl.slices), warps * 32, smem, st>>>(
            g, mask, all_cells, bin_start, bin_cnt, bin_flag, bin_pts, pts_xyz, pts_vf, keytab16, sd, tl, template_bins,
            c_max, nb_rec, nb_n, tie_cells, tie_count, n_template_cells, exact_cells);
        if (c_max == cand_cap) break;
        c_min = c_max;
        c_max = std::min(cand_cap, 3 * c_max);
    }
    return cudaGetLastError();
}
} // namespace hb
