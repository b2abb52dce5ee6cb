// Host stand-in for the CUDA runtime header, enough to compile the arithmetic headers of
// mdsm_gb300/csrc with a C++ compiler (built with -ffp-contract=off: one rounding an operation).
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#define __device__
#define __host__
#define __forceinline__ inline

static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline uint32_t __float_as_uint(float f)
{
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
}
static inline float __uint_as_float(uint32_t u)
{
    float f;
    memcpy(&f, &u, 4);
    return f;
}
static inline double __hiloint2double(int hi, int lo)
{
    const uint64_t u = (uint64_t)(uint32_t)hi << 32 | (uint32_t)lo;
    double d;
    memcpy(&d, &u, 8);
    return d;
}
