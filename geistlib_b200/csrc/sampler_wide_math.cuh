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

/*
 * (float) ((double) e / S), for quotients in the normal range. With 1 / S in two floats the remainder r = e / S - q of
 * q = fl(e * hi) is known to 1.5 * 2^-47 of the quotient. That decides the rounding unless the quotient lies so close to a
 * midpoint of two floats; r is then at least 2^-26 of it, and a 2^19-th of r covers the error: where q + r does not round
 * the same with that much less and more, the division has to decide (one quotient in 10^6).
 */
struct WideQuotient {
    double S;
    float  hi, lo; /* 2^62 / S: whole units of a mass, so that nothing has to be scaled behind them */
    __device__ __forceinline__ explicit WideQuotient(double s) : S(s) {
        const double inv = 0x1p62 / s;
        hi               = __double2float_rn(inv);
        lo               = __double2float_rn(inv - (double) hi);
    }
    /* 2^62 p in five FP32 operations; sets `unsure` where it may be the rounded quotient's neighbour */
    __device__ __forceinline__ float quick(float e, bool &unsure) const {
        const float q    = __fmul_rn(e, hi);
        const float r    = __fmaf_rn(e, lo, __fmaf_rn(e, hi, -q));
        const float less = __fmaf_rn(r, 1.0f - 0x1p-19f, q);
        unsure |= less != __fmaf_rn(r, 1.0f + 0x1p-19f, q);
        return less;
    }
    __device__ __forceinline__ float divide(float e) const { return __double2float_rn((double) e / S); }
    __device__ __forceinline__ float operator()(float e) const {
        bool        unsure = false;
        const float p      = quick(e, unsure) * 0x1p-62f;
        return unsure ? divide(e) : p;
    }
};

/* A probability in units of 2^-62, as the multi-pass path adds them up: a row's add up to less than 2^63, exactly down to
 * p = 2^-38 and in any order. */
__device__ __forceinline__ long long wide_mass(float p) { return __float2ll_rz(p * 0x1p62f); }
__device__ __forceinline__ double mass_value(long long m) { return (double) m * 0x1p-62; }

} /* namespace gb */
