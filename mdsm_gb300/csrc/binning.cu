// binning.cu -- time downsampling of channel-major blocks for downsampled DM passes.
//
// The reference downsamples with src/mdsm/dedispersion_kernel.cu:203-264 (mean of binsize
// samples, launched at src/mdsm/dedispersion_thread.cu:116-144) and the prototype
// src/prototypes/binner.cu:13-71 (sum / sqrt(binsize)), but both index the buffer as
// interleaved [t][c] while MDSM's blocks are channel-major [c][t], so passes with binsize > 1
// do not dedisperse the right samples there.  Here out[c][t] = f(sum_{k<b} in[c][t*b + k])
// on the channel-major layout, with f the plain sum (exact: integer samples widen to uint16 or
// int32), the mean, or sum / sqrt(b).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "internal.h"

namespace mdsm {

template <typename TIn, typename TOut>
__global__ void k_downsample(const TIn *__restrict__ in, long long in_stride, long long nout,
                             int b, int mode, float scale, TOut *__restrict__ out,
                             long long out_stride)
{
    const int c = blockIdx.y;
    const TIn *r = in + (size_t)c * in_stride;
    TOut *o = out + (size_t)c * out_stride;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nout;
         t += (long long)gridDim.x * blockDim.x) {
        const TIn *p = r + t * b;
        if (mode == 0) {
            long long acc = 0;
            double facc = 0.0;
            if (std::is_floating_point<TIn>::value) {
                for (int k = 0; k < b; ++k) facc = __dadd_rn(facc, (double)p[k]);
                o[t] = (TOut)facc;
            } else {
                for (int k = 0; k < b; ++k) acc += (long long)p[k];
                o[t] = (TOut)acc;
            }
        } else {
            float acc = 0.0f;
            for (int k = 0; k < b; ++k) acc = __fadd_rn(acc, (float)p[k]);
            o[t] = (TOut)__fmul_rn(acc, scale);
        }
    }
}

// The sum of B floats as the double sum above rounds it.  Two floats: the double sum's rounding to
// float is the float sum's.  More: where the exponents lie within 2^17 of one another the double
// sum is exact at every step, and so is the float sum with its errors added beside it (both are
// whole numbers of the smallest sample's last bit, within 24 bits), so the last addition rounds
// the exact sum once.  Double operations take a scheduler 64 clocks a warp: summing in double ran
// at 14 % of the copy rate.
template <int B>
__device__ __forceinline__ float sum_as_double(const float (&x)[B])
{
    if constexpr (B == 2) return __fadd_rn(__fadd_rn(0.0f, x[0]), x[1]);
    uint32_t hi = 0u, lo = 0x7f800000u;
#pragma unroll
    for (int k = 0; k < B; ++k) {
        const uint32_t e = __float_as_uint(x[k]) & 0x7f800000u;
        hi = max(hi, e);
        lo = min(lo, x[k] == 0.0f ? 0x7f800000u : e);
    }
    if (hi < (250u << 23) && lo > 0u && hi <= lo + (17u << 23)) {
        float s = 0.0f, err = 0.0f;
#pragma unroll
        for (int k = 0; k < B; ++k) {
            const float n = __fadd_rn(s, x[k]), bb = __fsub_rn(n, s);
            err = __fadd_rn(err, __fadd_rn(__fsub_rn(s, __fsub_rn(n, bb)), __fsub_rn(x[k], bb)));
            s = n;
        }
        return __fadd_rn(s, err);
    }
    double d = 0.0;
#pragma unroll
    for (int k = 0; k < B; ++k) d = __dadd_rn(d, (double)x[k]);
    return (float)d;
}

// Sums of B = 2, 4 or 8 samples on 16-byte aligned rows: a thread reads the samples of 16 bytes
// of output (or of 4 outputs) as 16-byte pieces.  Bound by DRAM: float 1024 x 2^15 by 2 and by 4 in
// 37 us each (83 and 72 % of the copy rate); one double sum a thread (FP64 pipe 86 %) took 490 together.
template <typename TIn, typename TOut, int B>
__global__ void __launch_bounds__(256)
    k_downsample_sum(const TIn *__restrict__ in, long long in_stride, long long nout,
                     TOut *__restrict__ out, long long out_stride)
{
    constexpr int NO = 16 / (int)sizeof(TOut);             // outputs of a thread
    constexpr int NI = NO * B;                             // samples it reads
    constexpr int NV = NI * (int)sizeof(TIn) / 4;          // words
    const TIn *r = in + (size_t)blockIdx.y * in_stride;
    TOut *o = out + (size_t)blockIdx.y * out_stride;
    for (long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * NO; t < nout;
         t += (long long)gridDim.x * blockDim.x * NO) {
        __align__(16) TIn x[NI];
        const bool whole = t + NO <= nout;
        if (whole) {
            const TIn *p = r + t * B;
            if constexpr (NV % 4 == 0) {
#pragma unroll
                for (int v = 0; v < NV / 4; ++v)
                    reinterpret_cast<uint4 *>(x)[v] = __ldg(reinterpret_cast<const uint4 *>(p) + v);
            } else {
                *reinterpret_cast<uint2 *>(x) = __ldg(reinterpret_cast<const uint2 *>(p));
            }
        } else {
#pragma unroll
            for (int k = 0; k < NI; ++k) x[k] = t + k / B < nout ? __ldg(r + t * B + k) : TIn(0);
        }
        __align__(16) TOut y[NO];
#pragma unroll
        for (int i = 0; i < NO; ++i) {
            if constexpr (std::is_same<TIn, float>::value) {
                float q[B];
#pragma unroll
                for (int k = 0; k < B; ++k) q[k] = x[i * B + k];
                y[i] = (TOut)sum_as_double<B>(q);
            } else {
                int acc = 0;
#pragma unroll
                for (int k = 0; k < B; ++k) acc += (int)x[i * B + k];
                y[i] = (TOut)acc;
            }
        }
        if (whole) {
            *reinterpret_cast<uint4 *>(o + t) = *reinterpret_cast<const uint4 *>(y);
        } else {
#pragma unroll
            for (int i = 0; i < NO; ++i)
                if (t + i < nout) o[t + i] = y[i];
        }
    }
}

template <typename TIn, typename TOut>
static void launch_ds(const void *in, long long in_stride, int nchans, long long nout, int b,
                      int mode, float scale, void *out, long long out_stride, cudaStream_t st)
{
    const bool aligned = (((uintptr_t)in | (uintptr_t)out |
                           (uintptr_t)(in_stride * (long long)sizeof(TIn)) |
                           (uintptr_t)(out_stride * (long long)sizeof(TOut))) & 15) == 0;
    if (mode == 0 && aligned && (b == 2 || b == 4 || b == 8)) {
        const long long per = 256 * 16 / (long long)sizeof(TOut);
        dim3 g((unsigned)std::min<long long>((nout + per - 1) / per, 1024), (unsigned)nchans);
        const TIn *i = static_cast<const TIn *>(in);
        TOut *o = static_cast<TOut *>(out);
        if (b == 2) k_downsample_sum<TIn, TOut, 2><<<g, 256, 0, st>>>(i, in_stride, nout, o, out_stride);
        else if (b == 4) k_downsample_sum<TIn, TOut, 4><<<g, 256, 0, st>>>(i, in_stride, nout, o, out_stride);
        else k_downsample_sum<TIn, TOut, 8><<<g, 256, 0, st>>>(i, in_stride, nout, o, out_stride);
        return;
    }
    dim3 grid((unsigned)std::min<long long>((nout + 255) / 256, 1024), (unsigned)nchans);
    k_downsample<TIn, TOut><<<grid, 256, 0, st>>>(static_cast<const TIn *>(in), in_stride, nout,
                                                  b, mode, scale, static_cast<TOut *>(out),
                                                  out_stride);
}

mdsm_status downsample(const void *in, int in_dtype, int nchans, long long in_stride,
                       long long len, int b, int mode, void *out, int out_dtype,
                       long long out_stride, cudaStream_t st)
{
    if (b < 1 || nchans <= 0 || len < 0) return fail(MDSM_EINVAL, "downsample: bad arguments");
    const long long nout = len / b;
    if (out_stride < nout) return fail(MDSM_ERANGE, "downsample: output pitch too small");
    if (nout == 0) return MDSM_OK;
    const float scale = mode == 1 ? 1.0f / (float)b : (mode == 2 ? 1.0f / sqrtf((float)b) : 1.0f);
    if (mode != 0 && out_dtype != MDSM_F32)
        return fail(MDSM_EINVAL, "downsample: mean and 1/sqrt(b) outputs are float32");
    if (mode == 0 && in_dtype == MDSM_U8 && out_dtype == MDSM_U16 && b > 257)
        return fail(MDSM_ERANGE, "downsample: uint16 sums hold at most 257 uint8 samples");
#define DS(TI, TO) launch_ds<TI, TO>(in, in_stride, nchans, nout, b, mode, scale, out, out_stride, st)
    if (in_dtype == MDSM_U8 && out_dtype == MDSM_U16) DS(uint8_t, uint16_t);
    else if (in_dtype == MDSM_U8 && out_dtype == MDSM_I32) DS(uint8_t, int32_t);
    else if (in_dtype == MDSM_U8 && out_dtype == MDSM_F32) DS(uint8_t, float);
    else if (in_dtype == MDSM_U16 && out_dtype == MDSM_I32) DS(uint16_t, int32_t);
    else if (in_dtype == MDSM_U16 && out_dtype == MDSM_F32) DS(uint16_t, float);
    else if (in_dtype == MDSM_I16 && out_dtype == MDSM_I32) DS(int16_t, int32_t);
    else if (in_dtype == MDSM_I16 && out_dtype == MDSM_F32) DS(int16_t, float);
    else if (in_dtype == MDSM_F32 && out_dtype == MDSM_F32) DS(float, float);
    else return fail(MDSM_EINVAL, "downsample: unsupported sample types");
#undef DS
    MDSM_CUDA_TRY(cudaGetLastError());
    return MDSM_OK;
}

}  // namespace mdsm

extern "C" mdsm_status mdsm_downsample_device(const void *d_in, int in_dtype, int nchans,
                                              long long in_stride, long long len, int binsize,
                                              int mode, void *d_out, int out_dtype,
                                              long long out_stride, void *stream)
{
    if (!d_in || !d_out) return mdsm::fail(MDSM_EINVAL, "null argument");
    return mdsm::downsample(d_in, in_dtype, nchans, in_stride, len, binsize, mode, d_out,
                            out_dtype, out_stride, static_cast<cudaStream_t>(stream));
}
