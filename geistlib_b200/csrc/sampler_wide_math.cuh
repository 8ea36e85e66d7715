/*
 * sampler_wide_math.cuh — the arithmetic of wide top-p rows. It gives what the multi-pass path's gives: a row must not come
 * out otherwise because of the path it took.
 */
#pragma once
#include "sampler_device.cuh"

namespace gb {

/*
 * expf as a correctly rounded one gives it, for a <= 0: 2^m * 2^(j/32) * e^r by Tang's table-driven scheme (P. Tang, ACM
 * TOMS 15, 1989) in double, the table one entry per lane (t32 = 2^(lane / 32)): all lanes of the warp call. r is at most
 * ln 2 / 64, where the series cut behind r^6 / 720 is good to 4e-18, so the value before its rounding to binary32 is as
 * good as exp()'s: exp_exact gives the same bits for every float from -0 to -130, on the device (the test does that). Every a
 * below -120 gives 0, as exp_exact does from -104 on. A NaN does not come back (the caller has excluded it).
 */
__device__ __forceinline__ float wide_exp(float a, double t32) {
    const double ad = (double) fmaxf(a, -120.0f);
    const double t  = __fma_rn(ad, 46.166241308446829, 0x1.8p52); /* 32 / ln 2; the addend leaves the nearest whole number in the low word */
    const int    n  = __double2loint(t);
    const double nd = t - 0x1.8p52;
    double       r  = __fma_rn(nd, -0x1.62e42fefa39efp-6, ad); /* ln 2 / 32 in two doubles */
    r               = __fma_rn(nd, -0x1.abc9e3b39803fp-61, r);
    double q        = __fma_rn(r, 1.0 / 720.0, 1.0 / 120.0);
    q               = __fma_rn(q, r, 1.0 / 24.0);
    q               = __fma_rn(q, r, 1.0 / 6.0);
    q               = __fma_rn(q, r, 0.5);
    q               = __fma_rn(q, r, 1.0);
    q               = q * r;
    const int    lo = __shfl_sync(0xffffffffu, __double2loint(t32), n); /* lane n modulo 32 */
    const int    hi = __shfl_sync(0xffffffffu, __double2hiint(t32), n) + ((n << 15) & (int) 0xfff00000);
    const double T  = __hiloint2double(hi, lo);
    return __double2float_rn(__fma_rn(T, q, T));
}

/* (float) (e / S): the quotient to 2^-47, then one rounding (inv_hi + inv_lo = 1 / S). None of 3e7 differed from the
 * rounded quotient of 64 bits. */
__device__ __forceinline__ float wide_prob(float e, float inv_hi, float inv_lo) {
    const float q = __fmul_rn(e, inv_hi);
    return __fadd_rn(q, __fmaf_rn(e, inv_lo, __fmaf_rn(e, inv_hi, -q)));
}

/* A probability in units of 2^-62, as the multi-pass path adds them up: a row's add up to less than 2^63, exactly down to
 * p = 2^-38 and in any order. */
__device__ __forceinline__ long long wide_mass(float p) { return __float2ll_rz(p * 0x1p62f); }
__device__ __forceinline__ double mass_value(long long m) { return (double) m * 0x1p-62; }

} /* namespace gb */
