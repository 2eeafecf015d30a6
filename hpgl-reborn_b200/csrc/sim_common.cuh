// Scalar maths shared by the simulation kernels (sgs.cu, sim_weights.cu).
#pragma once
#include <cuda_runtime.h>

namespace hb
{
// gaussian_cdf_t (gaussian_distribution.h): Abramowitz & Stegun 26.2.17 and the
// Odeh & Evans inverse, every operation rounded as the reference's double code
// rounds it (no contraction); exp and log are CUDA's (within 1 ulp of glibc's).
__device__ __forceinline__ double sgs_gauss_inverse(double pr, double mean, double var)
{
    if (pr <= 0.0 || pr >= 1.0) return mean;
    double p2 = pr > 0.5 ? __dsub_rn(1.0, pr) : pr;
    if (p2 < 1e-150) p2 = 1e-150;
    const double y = __dsqrt_rn(log(__ddiv_rn(1.0, __dmul_rn(p2, p2))));
    double num = __dadd_rn(__dmul_rn(-0.453642210148e-4, y), -0.0204231210245);
    num = __dadd_rn(__dmul_rn(num, y), -0.342242088547);
    num = __dadd_rn(__dmul_rn(num, y), -1.0);
    num = __dadd_rn(__dmul_rn(num, y), -0.322232431088);
    double den = __dadd_rn(__dmul_rn(0.38560700634e-2, y), 0.103537752850);
    den = __dadd_rn(__dmul_rn(den, y), 0.531103462366);
    den = __dadd_rn(__dmul_rn(den, y), 0.588581570495);
    den = __dadd_rn(__dmul_rn(den, y), 0.0993484626060);
    double xp = __dadd_rn(y, __ddiv_rn(num, den));
    if (pr < 0.5) xp = -xp;
    return __dadd_rn(__dmul_rn(xp, __dsqrt_rn(var)), mean);
}

// the correlogram scale of a mean (corellogramed_weights_3, my_kriging_weights.h:407-438)
__device__ __forceinline__ double sis_sigma(float mean)
{
    double m = (double)mean;
    if (m == 0) m = __dadd_rn(m, 0.00001);
    if (m == 1) m = __dsub_rn(m, 0.00001);
    return __dsqrt_rn(__dmul_rn(m, __dsub_rn(1.0, m)));
}
} // namespace hb
