// clip.cuh -- the RFI clip's rule as bounds in the sample type, shared by the standalone clip
// (rfi.cu) and the fused batched launch (dedisp.cu).
//
// A sample v is clipped when fabs(v - mean) >= lim, evaluated in double (the rounded difference
// is monotone in v), so on each side of the mean the test holds from some sample value outward:
// v is clipped exactly when v <= lo or v >= hi.  The bounds start from the real-valued estimates
// and are settled with the double test itself.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mdsm {

// Mean and sigma of n integer samples from their exact sums.
__device__ __forceinline__ void mean_sigma_ll(long long s1, long long s2, long long n, double *mu,
                                              double *sig)
{
    const double m = __ddiv_rn((double)s1, (double)n);
    const double var = __dadd_rn(__ddiv_rn((double)s2, (double)n), -__dmul_rn(m, m));
    *mu = m;
    *sig = var > 0.0 ? __dsqrt_rn(var) : 0.0;
}

__device__ __forceinline__ bool clip_test(double v, double mu, double lim)
{
    return fabs(__dadd_rn(v, -mu)) >= lim;
}

// Integer samples VMIN..VMAX: lo in [VMIN - 1, VMAX], hi in [VMIN, VMAX + 1], lo < hi.
template <int VMIN, int VMAX>
__device__ __forceinline__ void clip_bounds_int(double mu, double lim, int *lo, int *hi)
{
    *lo = VMIN - 1;
    *hi = VMAX + 1;
    if (!(lim >= 0.0)) return;  // (an infinite factor times sigma 0: nothing compares true)
    const int c = (int)ceil(mu);  // samples below c lie below the mean
    int h = (int)fmin(fmax(ceil(mu + lim), (double)c), (double)(VMAX + 1));
    while (h > c && clip_test((double)(h - 1), mu, lim)) --h;
    while (h <= VMAX && !clip_test((double)h, mu, lim)) ++h;
    int l = (int)fmax(fmin(floor(mu - lim), (double)(c - 1)), (double)(VMIN - 1));
    while (l < c - 1 && clip_test((double)(l + 1), mu, lim)) ++l;
    while (l >= VMIN && !clip_test((double)l, mu, lim)) --l;
    *lo = l;
    *hi = h;
}

// The mean as a sample VMIN..VMAX.
template <int VMIN, int VMAX>
__device__ __forceinline__ int clip_rep_int(double mu)
{
    return min(max(__double2int_rn(mu), VMIN), VMAX);
}

// Floats in order as unsigned keys (-inf lowest).
__device__ __forceinline__ uint32_t float_key(float f)
{
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Float samples: NaN for a side on which no sample is clipped (comparisons with it are false,
// as they are for a NaN sample).
__device__ __forceinline__ void clip_bounds_f32(double mu, double lim, float *lo, float *hi)
{
    const float none = __uint_as_float(0x7fffffffu);
    *lo = *hi = none;
    if (!(lim >= 0.0) || isnan(mu)) return;
    const uint32_t kc = float_key(__double2float_ru(mu));  // the smallest float at or above mu
    const uint32_t kinf = 0xff800000u, kninf = 0x007fffffu;
    auto test = [&](uint32_t k) { return clip_test((double)key_float(k), mu, lim); };
    if (test(kinf)) {  // the smallest key in [kc, kinf] that is clipped
        uint32_t h = float_key(__double2float_ru(mu + lim));
        h = min(max(h, kc), kinf);
        if (!test(h) || (h > kc && test(h - 1))) {
            uint32_t a = kc, b = kinf;  // (test(b) holds)
            while (a < b) {
                const uint32_t m = a + (b - a) / 2;
                if (test(m)) b = m;
                else a = m + 1;
            }
            h = a;
        }
        *hi = key_float(h);
    }
    if (kc > kninf && test(kninf)) {  // the largest key in [kninf, kc) that is clipped
        uint32_t l = float_key(__double2float_rd(mu - lim));
        l = max(min(l, kc - 1), kninf);
        if (!test(l) || (l < kc - 1 && test(l + 1))) {
            uint32_t a = kninf, b = kc - 1;  // (test(a) holds)
            while (a < b) {
                const uint32_t m = b - (b - a) / 2;
                if (test(m)) a = m;
                else b = m - 1;
            }
            l = a;
        }
        *lo = key_float(l);
    }
}

}  // namespace mdsm
