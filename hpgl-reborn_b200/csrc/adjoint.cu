// Leave-one-out ordinary kriging of the conditioning points and its adjoint.
//
// No counterpart in the reference (HPGL has no cross-validation and no
// gradients). For every target point i the system is the reference's OK system
// (my_kriging_weights.h:198-361): A[r][c] = C(p_r - p_c), b[r] = C(p_r - p_i),
// x = A^-1 b, y = A^-1 1, mu = (sum x - 1) / sum y, lambda = x - mu y and the
// estimate zhat_i = lambda . z over the neighbours (combiner.h:10-25 with mean 0).
//
// The covariance is evaluated in FP64 from M = diag(1/r0, 1/r1, 1/r2) R, the
// reference's transform divided by ranges[0] (cov_model.h:16-61): u = |M v|,
// C = sill for r0 u < 1e-4, else (sill - nugget) f(u) with
//   spherical   f = 1 - 1.5 u + 0.5 u^3 (u <= 1), 0 beyond
//   exponential f = exp(-3 u)
//   Gaussian    f = exp(-3 u^2)                        (cov_model.h:146-183).
//
// Adjoint. With K = [A 1; 1^T 0] symmetric, zhat = [z; 0]^T K^-1 [b; 1], so
//   d zhat = alpha^T db - alpha^T dA lambda,   d zhat / d z = lambda,
// where [alpha; beta] = K^-1 [z; 0]: alpha = A^-1 z - beta A^-1 1,
// beta = (1^T A^-1 z) / (1^T A^-1 1). The backward kernel recomputes the factor
// (nothing is stored between the passes), forms alpha and lambda, and sums the
// covariance derivatives of every b and A entry weighted by alpha_r and
// -alpha_r lambda_c:
//   dC/dsill = f, dC/dnugget = -f, dC/dM_ab = (sill - nugget) f'(u) (M v)_a v_b / u
// (dC/dsill = 1 and the rest 0 on the C(0) branch). The host maps dM to ranges
// and angles.
//
// One warp per target (neighbour counts up to 32): the covariances block by block
// of the lower triangle in the layout of the FP64 tensor instruction, its
// factorisation with the three right-hand sides, and the back substitution of
// warp64.cuh. The derivative sums run over the same blocks, an entry and its
// mirror together, and d zhat / dM = M S with S_bc = sum (.) v_b v_c, which is
// symmetric: six sums a lane in place of nine, added up over a warp's targets
// and then a block's before the 11 atomic additions.
//
// What bounds it: the chain of pivots and the covariances' exponentials, at 27
// targets an SM. Measured at 4,000 targets of 24 neighbours, Gaussian: forward
// 87 us with a lane a row (which evaluated every entry of a 32-wide padded
// triangle with half its lanes idle), 23.6 us now; adjoint 138 and 38.4 us (44.6
// in five blocks of 96 registers on an SM, which spill its sums).
#include "../../include/hpgl_b200.h"
#include "engine_api.h"
#include "warp64.cuh"

#include <cuda_runtime.h>

#include <cstdint>
#include <string>

namespace hb
{
namespace
{
constexpr int kLooWarps = 4;  // warps (targets) per block
constexpr int kLooBlocks = 5;     // blocks on an SM, forward: 20 warps of 96 registers
constexpr int kAdjointBlocks = 4; // adjoint: its sums take 16 registers more

// the variogram
struct LooModel
{
    double M[9];
    double r0, sill, nugget;
};

struct LooParams
{
    const int *pts_xyz; // 3 ints per point
    const double *values;
    int n_pts;
    const int *targets;
    const int *nb_idx; // k point ids per target
    const int *nb_cnt;
    int n_targets;
    int k;
    int cov_type;
    LooModel model;                    // M, sill and nugget as host values, or
    const double *M, *sill, *nugget;   // (M set) where they are on the device
};

// the block's copy of the variogram
__device__ __forceinline__ void load_model(const LooParams &P, LooModel &m)
{
    double *d = reinterpret_cast<double *>(&m);
    const int i = threadIdx.x;
    if (i < 12) d[i] = reinterpret_cast<const double *>(&P.model)[i];
    if (P.M)
    {
        if (i < 9) d[i] = P.M[i];
        if (i == 10) d[i] = *P.sill;
        if (i == 11) d[i] = *P.nugget;
    }
    __syncthreads();
}

struct CovD
{
    double c;     // covariance
    double f;     // dC/dsill (and -dC/dnugget)
    double gu;    // (sill - nugget) f'(u) / u: dC/dM_ab = gu (M v)_a v_b
    bool at_zero; // the C(0) branch
};

__device__ __forceinline__ CovD cov_d(const LooModel &P, int cov_type, int dx, int dy, int dz)
{
    CovD o;
    const double v0 = (double)dx, v1 = (double)dy, v2 = (double)dz;
    const double w0 = P.M[0] * v0 + P.M[1] * v1 + P.M[2] * v2;
    const double w1 = P.M[3] * v0 + P.M[4] * v1 + P.M[5] * v2;
    const double w2 = P.M[6] * v0 + P.M[7] * v1 + P.M[8] * v2;
    const double u = sqrt(w0 * w0 + w1 * w1 + w2 * w2);
    o.at_zero = P.r0 * u < 0.0001;
    if (o.at_zero)
    {
        o.c = P.sill;
        o.f = 0.0;
        o.gu = 0.0;
        return o;
    }
    const double s = P.sill - P.nugget;
    double f, fp;
    if (cov_type == 1)
    {
        f = exp(-3.0 * u);
        fp = -3.0 * f;
    }
    else if (cov_type == 2)
    {
        f = exp(-3.0 * u * u);
        fp = -6.0 * u * f;
    }
    else if (u > 1.0)
    {
        f = 0.0;
        fp = 0.0;
    }
    else
    {
        f = 1.0 - 1.5 * u + 0.5 * u * u * u;
        fp = -1.5 + 1.5 * u * u;
    }
    o.c = s * f;
    o.f = f;
    o.gu = s * fp / u;
    return o;
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// one warp's shared memory
struct LooSmem
{
    WarpSmem<3, false> T;
    int4 pt[kWarpN]; // the neighbours' coordinates
};

// Everything one target's forward pass leaves in registers.
struct LooSolve
{
    int n;
    bool ok;
    int pid;        // this lane's neighbour, -1 for padding rows
    int at;         // its place among the unknowns
    int px, py, pz; // its coordinates
    int tx, ty, tz; // the target's
    double lambda;  // OK weight
    double alpha;   // adjoint weight
    double zhat;
};

// Assemble, factor and solve the target's system; lane r holds neighbour r.
__device__ LooSolve loo_solve(const LooParams &P, const LooModel &m, int t, LooSmem &W)
{
    const int lane = threadIdx.x & 31;
    LooSolve S;
    S.n = min(P.nb_cnt[t], P.k);
    const int n = S.n, nb = (n + 7) >> 3;
    const bool live = lane < n;
    S.pid = live ? P.nb_idx[(long long)t * P.k + lane] : -1;
    const int tp = P.targets[t];
    S.tx = P.pts_xyz[3 * tp];
    S.ty = P.pts_xyz[3 * tp + 1];
    S.tz = P.pts_xyz[3 * tp + 2];
    S.px = live ? P.pts_xyz[3 * S.pid] : 0;
    S.py = live ? P.pts_xyz[3 * S.pid + 1] : 0;
    S.pz = live ? P.pts_xyz[3 * S.pid + 2] : 0;
    const double z = live ? P.values[S.pid] : 0.0;
    const double b = live ? cov_d(m, P.cov_type, S.px - S.tx, S.py - S.ty, S.pz - S.tz).c : 0.0;
    S.at = mma_slot(lane, n, nb);
    __syncwarp(); // the previous target's reads are done
    W.pt[S.at] = make_int4(S.px, S.py, S.pz, 0);
    W.T.y[0][S.at] = b;
    W.T.y[1][S.at] = live ? 1.0 : 0.0;
    W.T.y[2][S.at] = z;
    __syncwarp();

    // the lower triangle's blocks (the diagonal ones whole), padding rows identity
    const int r = lane >> 2, q = lane & 3, at = blk_chunk(r, q);
    double2 *LM = reinterpret_cast<double2 *>(W.T.LM);
    int blk = 0;
#pragma unroll 1
    for (int i = 0; i < nb; ++i)
    {
        const int row = 8 * i + r;
        const int4 a = W.pt[row];
#pragma unroll 1
        for (int k = 0; k <= i; ++k, ++blk)
        {
            double e[2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const int col = 8 * k + 2 * q + h;
                const int4 c = W.pt[col];
                e[h] = row == col ? 1.0 : 0.0;
                if (row < n && col < n) e[h] = cov_d(m, P.cov_type, a.x - c.x, a.y - c.y, a.z - c.z).c;
            }
            LM[blk * 32 + at] = make_double2(e[0], e[1]); // read back by this lane alone
        }
    }
    Blk A[1][kWarpBlocks];
#pragma unroll
    for (int i = 0; i < kWarpNB; ++i)
    {
        if (i >= nb) break;
#pragma unroll
        for (int k = 0; k <= i; ++k)
        {
            const double2 v = LM[blk_at(i, k) * 32 + at];
            A[0][blk_at(i, k)] = Blk{v.x, v.y};
        }
    }
    // L y = [b, 1, z], then L^T x = y
    const bool fail = warp_eliminate<3, false, false, true>(W.T, lane, nb, A);
    warp_back<3>(W.T, lane, nb);
    const double x0 = live ? W.T.y[0][S.at] : 0.0, x1 = live ? W.T.y[1][S.at] : 0.0, x2 = live ? W.T.y[2][S.at] : 0.0;
    const double sx = warp_sum(x0), sy = warp_sum(x1), sz = warp_sum(x2);
    const double mu = (sx - 1.0) / sy, beta = sz / sy;
    S.lambda = live ? x0 - mu * x1 : 0.0;
    S.alpha = live ? x2 - beta * x1 : 0.0;
    S.zhat = warp_sum(S.lambda * z);
    S.ok = n > 0 && !fail && !(fabs(sy) < 1e-15) && S.zhat == S.zhat;
    return S;
}

__global__ void __launch_bounds__(32 * kLooWarps, kLooBlocks) k_loo_forward(const LooParams P, double *__restrict__ zhat,
                                                                           signed char *__restrict__ status)
{
    __shared__ LooSmem sm[kLooWarps];
    __shared__ LooModel m;
    load_model(P, m);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int t = blockIdx.x * kLooWarps + warp; t < P.n_targets; t += gridDim.x * kLooWarps)
    {
        const LooSolve S = loo_solve(P, m, t, sm[warp]);
        if (lane == 0)
        {
            zhat[t] = S.ok ? S.zhat : 0.0;
            if (status) status[t] = S.ok ? 0 : (S.n == 0 ? 1 : 2);
        }
    }
}

// grad_values[p] += g lambda; grad_params[0..8] += g dzhat/dM, [9] sill, [10] nugget.
__global__ void __launch_bounds__(32 * kLooWarps, kAdjointBlocks) k_loo_adjoint(const LooParams P,
                                                                           const double *__restrict__ g_zhat,
                                                                           double *__restrict__ grad_values,
                                                                           double *__restrict__ grad_params)
{
    __shared__ LooSmem sm[kLooWarps];
    __shared__ LooModel m;
    __shared__ double part[kLooWarps][8];
    load_model(P, m);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    LooSmem &W = sm[warp];
    // sums over the warp's targets: wgt f, wgt on the C(0) branch, and wgt gu v_b v_c
    double gf = 0.0, gz = 0.0, s6[6] = {0, 0, 0, 0, 0, 0};
    auto add = [&](int dx, int dy, int dz, double wgt) {
        const CovD d = cov_d(m, P.cov_type, dx, dy, dz);
        if (d.at_zero)
        {
            gz += wgt;
            return;
        }
        gf += wgt * d.f;
        const double v0 = (double)dx, v1 = (double)dy, v2 = (double)dz, h = wgt * d.gu;
        const double h0 = h * v0, h1 = h * v1, h2 = h * v2;
        s6[0] += h0 * v0;
        s6[1] += h0 * v1;
        s6[2] += h0 * v2;
        s6[3] += h1 * v1;
        s6[4] += h1 * v2;
        s6[5] += h2 * v2;
    };
    for (int t = blockIdx.x * kLooWarps + warp; t < P.n_targets; t += gridDim.x * kLooWarps)
    {
        const double g = g_zhat[t];
        if (g == 0.0) continue; // warp-uniform
        const LooSolve S = loo_solve(P, m, t, W);
        if (!S.ok) continue; // failed targets carry no gradient (warp-uniform)
        const bool live = lane < S.n;
        if (live) atomicAdd(&grad_values[S.pid], g * S.lambda);
        const double ga = g * S.alpha; // 0 beyond n
        __syncwarp();
        W.T.y[0][S.at] = S.lambda;
        W.T.y[1][S.at] = ga;
        __syncwarp();
        // alpha_r dC(b_r) - alpha_r sum_c lambda_c dC(A_rc), A_rc and A_cr together
        if (live) add(S.px - S.tx, S.py - S.ty, S.pz - S.tz, ga);
        const int r = lane >> 2, q = lane & 3, nb = (S.n + 7) >> 3;
#pragma unroll 1
        for (int i = 0; i < nb; ++i)
        {
            const int row = 8 * i + r;
            const int4 a = W.pt[row];
            const double lr = W.T.y[0][row], ar = W.T.y[1][row];
#pragma unroll 1
            for (int k = 0; k <= i; ++k)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    const int col = 8 * k + 2 * q + h;
                    const int4 c = W.pt[col];
                    const double lc = W.T.y[0][col], ac = W.T.y[1][col];
                    if (row < S.n && col < S.n)
                        add(a.x - c.x, a.y - c.y, a.z - c.z, k == i ? -ar * lc : -(ar * lc + ac * lr));
                }
        }
    }
    const double v[8] = {gf, gz, s6[0], s6[1], s6[2], s6[3], s6[4], s6[5]};
#pragma unroll
    for (int i = 0; i < 8; ++i)
    {
        const double s = warp_sum(v[i]);
        if (lane == 0) part[warp][i] = s;
    }
    __syncthreads();
    if (threadIdx.x < 11)
    {
        auto total = [&](int i) {
            double s = 0.0;
            for (int w = 0; w < kLooWarps; ++w) s += part[w][i];
            return s;
        };
        const int i = threadIdx.x;
        double s;
        if (i < 9)
        {
            const int a = i / 3, c = i % 3; // M S: S's entries (0, c), (1, c), (2, c)
            s = m.M[3 * a] * total(2 + c) + m.M[3 * a + 1] * total(c == 0 ? 3 : 4 + c) +
                m.M[3 * a + 2] * total(c == 0 ? 4 : 5 + c);
        }
        else
            s = i == 9 ? total(0) + total(1) : -total(0);
        atomicAdd(&grad_params[i], s);
    }
}

int fill_params(LooParams &P, const int *pts_xyz, const double *values, int n_pts, const int *targets,
                 const int *nb_idx, const int *nb_cnt, int n_targets, int k, int cov_type, const double *M, double r0,
                 const double *sill, const double *nugget, bool on_device)
{
    if (!sill || !nugget || !pts_xyz || !values || !targets || !nb_idx || !nb_cnt || !M || n_pts < 0 || n_targets < 0)
    {
        set_error("loo kriging: null array argument or negative size");
        return HPGL_B200_EINVAL;
    }
    if (k < 1)
    {
        set_error("loo kriging: max_neighbours must be >= 1");
        return HPGL_B200_EINVAL;
    }
    if (k > 32)
    {
        set_error("loo kriging: at most 32 neighbours per target are supported");
        return HPGL_B200_ELIMIT;
    }
    if (cov_type < 0 || cov_type > 2)
    {
        set_error("loo kriging: unknown covariance type");
        return HPGL_B200_EINVAL;
    }
    if (!(r0 > 0.0))
    {
        set_error("loo kriging: ranges[0] must be positive");
        return HPGL_B200_EINVAL;
    }
    P.pts_xyz = pts_xyz;
    P.values = values;
    P.n_pts = n_pts;
    P.targets = targets;
    P.nb_idx = nb_idx;
    P.nb_cnt = nb_cnt;
    P.n_targets = n_targets;
    P.k = k;
    P.cov_type = cov_type;
    P.model = LooModel{{}, r0, 0.0, 0.0};
    P.M = P.sill = P.nugget = nullptr;
    if (on_device)
    {
        P.M = M;
        P.sill = sill;
        P.nugget = nugget;
    }
    else
    {
        for (int i = 0; i < 9; ++i) P.model.M[i] = M[i];
        P.model.sill = *sill;
        P.model.nugget = *nugget;
    }
    return HPGL_B200_OK;
}

int grid_for(int n_targets, int blocks)
{
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long want = ((long long)n_targets + kLooWarps - 1) / kLooWarps;
    const long long cap = (long long)sms * blocks;
    return (int)(want < cap ? (want > 0 ? want : 1) : cap);
}

int loo_forward(const LooParams &P, double *zhat, signed char *status, void *stream)
{
    if (!zhat)
    {
        set_error("loo kriging: null output");
        return HPGL_B200_EINVAL;
    }
    if (P.n_targets == 0) return HPGL_B200_OK;
    k_loo_forward<<<grid_for(P.n_targets, kLooBlocks), 32 * kLooWarps, 0, (cudaStream_t)stream>>>(P, zhat, status);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
    {
        set_error(std::string("loo kriging: ") + cudaGetErrorString(e));
        return HPGL_B200_ECUDA;
    }
    return HPGL_B200_OK;
}

int loo_adjoint(const LooParams &P, const double *grad_zhat, double *grad_values, double *grad_params, void *stream)
{
    if (!grad_zhat || !grad_values || !grad_params)
    {
        set_error("loo kriging adjoint: null gradient argument");
        return HPGL_B200_EINVAL;
    }
    if (P.n_targets == 0) return HPGL_B200_OK;
    k_loo_adjoint<<<grid_for(P.n_targets, kAdjointBlocks), 32 * kLooWarps, 0, (cudaStream_t)stream>>>(P, grad_zhat, grad_values,
                                                                                      grad_params);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
    {
        set_error(std::string("loo kriging adjoint: ") + cudaGetErrorString(e));
        return HPGL_B200_ECUDA;
    }
    return HPGL_B200_OK;
}
} // namespace
} // namespace hb

extern "C" int hpgl_b200_loo_ok(const int *pts_xyz, const double *values, int n_pts, const int *targets, const int *nb_idx,
    const int *nb_cnt, int n_targets, int k, int cov_type, const double *M, double r0, double sill, double nugget, double *zhat, signed char *status, void *stream)
{
    hb::LooParams P;
    const int rc = hb::fill_params(P, pts_xyz, values, n_pts, targets, nb_idx, nb_cnt, n_targets, k, cov_type, M, r0,
                                   &sill, &nugget, false);
    return rc != HPGL_B200_OK ? rc : hb::loo_forward(P, zhat, status, stream);
}

extern "C" int hpgl_b200_loo_ok_adjoint(const int *pts_xyz, const double *values, int n_pts, const int *targets, const int *nb_idx,
    const int *nb_cnt, int n_targets, int k, int cov_type, const double *M, double r0, double sill, double nugget, const double *grad_zhat, double *grad_values, double *grad_params, void *stream)
{
    hb::LooParams P;
    const int rc = hb::fill_params(P, pts_xyz, values, n_pts, targets, nb_idx, nb_cnt, n_targets, k, cov_type, M, r0,
                                   &sill, &nugget, false);
    return rc != HPGL_B200_OK ? rc : hb::loo_adjoint(P, grad_zhat, grad_values, grad_params, stream);
}

extern "C" int hpgl_b200_loo_ok_device(const int *pts_xyz, const double *values, int n_pts, const int *targets, const int *nb_idx,
    const int *nb_cnt, int n_targets, int k, int cov_type, const double *M, double r0, const double *sill, const double *nugget, double *zhat, signed char *status, void *stream)
{
    hb::LooParams P;
    const int rc = hb::fill_params(P, pts_xyz, values, n_pts, targets, nb_idx, nb_cnt, n_targets, k, cov_type, M, r0,
                                   sill, nugget, true);
    return rc != HPGL_B200_OK ? rc : hb::loo_forward(P, zhat, status, stream);
}

extern "C" int hpgl_b200_loo_ok_adjoint_device(const int *pts_xyz, const double *values, int n_pts, const int *targets, const int *nb_idx,
    const int *nb_cnt, int n_targets, int k, int cov_type, const double *M, double r0, const double *sill, const double *nugget, const double *grad_zhat, double *grad_values, double *grad_params, void *stream)
{
    hb::LooParams P;
    const int rc = hb::fill_params(P, pts_xyz, values, n_pts, targets, nb_idx, nb_cnt, n_targets, k, cov_type, M, r0,
                                   sill, nugget, true);
    return rc != HPGL_B200_OK ? rc : hb::loo_adjoint(P, grad_zhat, grad_values, grad_params, stream);
}
