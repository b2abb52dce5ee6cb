// cutsum.cuh -- exact sums of floats by float operations, where a left-to-right double sum rounds
// nothing (the statistics of rfi.cu and detect.cu are defined by such sums, and a double operation
// takes a scheduler of this GPU 64 clocks a warp).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mdsm {

// A normal float as a double by integer operations (the conversion instruction runs at the
// double rate); `special` when the exponent field is 0 or 255.
__device__ __forceinline__ double float_bits_double(uint32_t b)
{
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)),
                            (int)(b << 29));
}
__device__ __forceinline__ uint32_t special_key(float x)
{
    return (__float_as_uint(x) & 0x7f800000u) - 0x00800000u;  // >= 0x7f000000: special
}

// The sum of a run of at most 1024 floats, where the left-to-right double sum rounds nothing: a
// float is cut at three fixed places, and each third is added exactly in float.  With E the
// exponent of a typical large sample, the thirds are whole multiples of u1 = 2^(E-11), u2 =
// 2^(E-26) and u3 = 2^(E-41); cutting with a constant C = 1.5 * 2^23 units rounds to the unit
// (for a sample below 2^22 of the first), so the second and third hold at most half a unit of
// the one before (1024 of them stay within 2^24 units: exact adds), and the first is watched.
// What a rare small sample leaves past the third is added exactly beside them, and its lowest bit
// noted (it is looked for in the bits of what each sample leaves: a float sum of those would absorb
// the smaller ones).  While the first's sums stay below 2^23 u1, and with what the others can hold
// (512 u1 and less) below 2^53 lowest bits, every partial sum is a whole number of lowest bits below
// 2^53: the double sum is exact at every step, in any order.  Otherwise (ok() false) the caller sums
// in double.  15 float operations a sample
// against one at the double rate (64 clocks of a scheduler for a warp).
struct CutSum {
    float c1, c2, c3, a1, a2, a3, a4, top, unit;
    __device__ __forceinline__ void start(float biggest)
    {
        // 2^E as a float, 0 (no cut fits) for zero, tiny, huge or special values
        const uint32_t e = __float_as_uint(biggest) & 0x7f800000u;
        const float p = e > (100u << 23) && e < (160u << 23) ? __uint_as_float(e) : 0.0f;
        c1 = p * 6144.0f;            // 1.5 * 2^(23 + E - 11)
        c2 = p * (1.5f / 8.0f);      // 1.5 * 2^(23 + E - 26)
        c3 = p * (1.5f / 262144.0f); // 1.5 * 2^(23 + E - 41)
        unit = c3 * (1.0f / 12582912.0f);
        a1 = a2 = a3 = a4 = top = 0.0f;
    }
    // the thirds of x; returns what is left past them
    __device__ __forceinline__ float cut(float x, float &h1, float &h2, float &h3) const
    {
        h1 = __fsub_rn(__fadd_rn(x, c1), c1);
        const float r1 = __fsub_rn(x, h1);
        h2 = __fsub_rn(__fadd_rn(r1, c2), c2);
        const float r2 = __fsub_rn(r1, h2);
        h3 = __fsub_rn(__fadd_rn(r2, c3), c3);
        return __fsub_rn(r2, h3);
    }
    template <int U>
    __device__ __forceinline__ void add(const float (&v)[U])
    {
        uint32_t left = 0u;
#pragma unroll
        for (int j = 0; j < U; ++j) {
            float h1, h2, h3;
            left |= __float_as_uint(cut(v[j], h1, h2, h3));
            a1 = __fadd_rn(a1, h1);
            a2 = __fadd_rn(a2, h2);
            a3 = __fadd_rn(a3, h3);
            top = fmaxf(top, fmaxf(fabsf(a1), __fadd_rn(fabsf(v[j]), fabsf(v[j]))));
        }
        if ((left & 0x7fffffffu) == 0u) return;  // (-0 leaves -0)
        // some sample of these left a part past the third (or is not finite, and leaves a NaN)
#pragma unroll 1
        for (int j = 0; j < U; ++j) {
            float x = v[0];
#pragma unroll
            for (int q = 1; q < U; ++q) x = j == q ? v[q] : x;
            float h1, h2, h3;
            const float r3 = cut(x, h1, h2, h3);
            if (r3 == 0.0f) continue;
            const float s = __fadd_rn(a4, r3), bb = __fsub_rn(s, a4);
            const float err = __fadd_rn(__fsub_rn(a4, __fsub_rn(s, bb)), __fsub_rn(r3, bb));
            const uint32_t b = __float_as_uint(x), m = (b & 0x7fffffu) | 0x800000u;
            // the lowest bit of x: 2^(e - 150) times the lowest set bit of its significand
            const float low = __fmul_rn(__uint_as_float(b & 0x7f800000u),
                                        __fmul_rn((float)(m & (0u - m)), 1.0f / 8388608.0f));
            unit = err == 0.0f && low > 0.0f ? fminf(unit, low) : 0.0f;
            a4 = s;
        }
    }
    __device__ __forceinline__ bool finite() const { return a1 == a1 && top < INFINITY; }
    __device__ __forceinline__ bool ok() const
    {
        // a partial sum: the first third's (at most top), 1024 halves of u1, of u2 and of u3 (513 u1)
        const float most = __fadd_rn(top, c1 * (513.0f / 12582912.0f));
        // (2^53 lowest bits as 2^29 of them times 2^24; NaN and infinities fail a comparison)
        return c1 > 0.0f && finite() && top < c1 * 0.66f &&
               most * (1.01f / 536870912.0f) < unit * 16777216.0f;
    }
    __device__ __forceinline__ double sum() const
    {
        return __dadd_rn(__dadd_rn(__dadd_rn((double)a1, (double)a2), (double)a3), (double)a4);
    }
};

}  // namespace mdsm
