// rfi.cu -- RFI clipping of a channel-major filterbank block, in place on the device.
//
// src/prototypes/rfi_clipper.cu:8-67 clips each row: mean and sigma over the row, then samples
// with |x - mean| >= 4 sigma are replaced by the mean.  Here the same rule runs per channel
// (over time) and then per spectrum (over channels at one time sample).  Two defects of the
// prototype are not reproduced: its accumulators start uninitialised (:33) and it also clips
// |x - mean| <= sigma/4 (:61).  Statistics are exact for integer samples (int64 sums) and use
// a fixed left-to-right order of double sums for float samples, so the device result equals
// the oracle's bit for bit.
//
// The double operations of the clip test are the slow pipe of this GPU (2 lanes per clock per
// SM), so a row's test is turned once into two bounds of the sample type (clip.cuh) and the
// samples are compared as integers or floats; the float statistics keep one double operation a
// sample, the multiply-add of the squares (FP64 pipe 56-59 % busy: what bounds them), and sum the
// samples themselves exactly in float (cutsum.cuh).
// uint8 4096 x 97921: 138 us the channels, 252 the spectra; before, with the test in double and one
// thread a spectrum, 2330 and 3003.  Float 1001 x 40003: 230 and 145 us; before 662 and 976.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>
#include <utility>

#include "clip.cuh"
#include "cutsum.cuh"
#include "internal.h"

namespace mdsm {

namespace cg = cooperative_groups;

namespace {

template <typename T>
struct Range;
template <>
struct Range<uint8_t> {
    static constexpr int lo = 0, hi = 255;
};
template <>
struct Range<uint16_t> {
    static constexpr int lo = 0, hi = 65535;
};
template <>
struct Range<int16_t> {
    static constexpr int lo = -32768, hi = 32767;
};

struct IntClip {
    int lo, hi, rep;  // v <= lo or v >= hi is replaced by rep
};

template <typename T>
__device__ __forceinline__ IntClip int_clip(long long s1, long long s2, long long n, double k)
{
    double mu, sig;
    mean_sigma_ll(s1, s2, n, &mu, &sig);
    IntClip c;
    clip_bounds_int<Range<T>::lo, Range<T>::hi>(mu, __dmul_rn(k, sig), &c.lo, &c.hi);
    c.rep = clip_rep_int<Range<T>::lo, Range<T>::hi>(mu);
    return c;
}

// The samples of one 32-bit word: SPW samples, sample e in bits [e * 8 * size, ...).
template <typename T>
__device__ __forceinline__ int word_sample(uint32_t w, int e)
{
    if constexpr (sizeof(T) == 1)
        return (int)((w >> (8 * e)) & 0xffu);
    else if constexpr (std::is_same<T, int16_t>::value)
        return (int)(int16_t)(w >> (16 * e));
    else
        return (int)((w >> (16 * e)) & 0xffffu);
}

// Bounds of a word's samples, ready to test the word (each sample its own bounds).
// uint8: the even and odd bytes as 16-bit lanes; a lane x plus 256 - b has bit 8 set when
// x >= b, so one 32-bit add tests two samples against a bound each.
template <typename T>
struct WordClip {
    IntClip c[2];
    __device__ __forceinline__ void set(const IntClip *s)
    {
        c[0] = s[0];
        c[1] = s[1];
    }
    // w with its clipped samples replaced
    __device__ __forceinline__ uint32_t apply(uint32_t w) const
    {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int v = word_sample<T>(w, e);
            if (v <= c[e].lo || v >= c[e].hi)
                w = (w & ~(0xffffu << (16 * e))) | ((uint32_t)(uint16_t)c[e].rep << (16 * e));
        }
        return w;
    }
};
template <>
struct WordClip<uint8_t> {
    uint32_t in_e, out_e, in_o, out_o, rep;
    __device__ __forceinline__ void set(const IntClip *s)
    {
        auto lanes = [](int a, int b) { return (uint32_t)(256 - a) | ((uint32_t)(256 - b) << 16); };
        in_e = lanes(s[0].lo + 1, s[2].lo + 1);
        out_e = lanes(s[0].hi, s[2].hi);
        in_o = lanes(s[1].lo + 1, s[3].lo + 1);
        out_o = lanes(s[1].hi, s[3].hi);
        rep = (uint32_t)s[0].rep | ((uint32_t)s[1].rep << 8) | ((uint32_t)s[2].rep << 16) |
              ((uint32_t)s[3].rep << 24);
    }
    __device__ __forceinline__ uint32_t apply(uint32_t w) const
    {
        const uint32_t e = w & 0x00ff00ffu, o = __byte_perm(w, 0u, 0x4341);
        const uint32_t be = ((e + out_e) | ~(e + in_e)) & 0x01000100u;
        const uint32_t bo = ((o + out_o) | ~(o + in_o)) & 0x01000100u;
        if ((be | bo) == 0u) return w;
        const uint32_t m = (be >> 8) * 0xffu | bo * 0xffu;
        return (w & ~m) | (rep & m);
    }
};

// Sums of a word's samples and of their squares (32-bit s1; s2 as wide as the caller's).
template <typename T>
__device__ __forceinline__ void word_sums(uint32_t w, int &s1, unsigned long long &s2)
{
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int v = word_sample<T>(w, e);
        s1 += v;
        s2 += (unsigned long long)((uint32_t)v * (uint32_t)v);  // (|v| < 2^16: 32 bits hold it)
    }
}

constexpr int kChanThreads = 512;

// One CTA per channel: exact statistics over the row, then the clip.  The row is read twice in
// 16-byte vectors (dp4a sums for uint8); the second read comes from L2 (the rows in flight are
// far below its size), so the DRAM traffic is one read plus the vectors that change.  On uint8
// 4096 ch x 97921 this replaced one byte a thread and three double operations a sample.
template <typename T>
__global__ void __launch_bounds__(kChanThreads, 4)
    k_clip_channels_int(T *__restrict__ x, long long stride, long long len, double k)
{
    constexpr int N = 16 / (int)sizeof(T);
    T *row = x + (size_t)blockIdx.x * stride;
    const int tid = threadIdx.x;
    // samples before the first 16-byte boundary, whole vectors, the rest
    const long long head =
        min(len, (long long)(((16 - ((uintptr_t)row & 15)) & 15) / sizeof(T)));
    uint4 *vec = reinterpret_cast<uint4 *>(row + head);
    const long long nv = (len - head) / N, tail = head + nv * N;
    long long a1 = 0;
    unsigned long long a2 = 0;
    auto one = [&](long long i) {
        const long long v = row[i];
        a1 += v;
        a2 += (unsigned long long)(v * v);
    };
    for (long long i = tid; i < head; i += kChanThreads) one(i);
    for (long long i = tail + tid; i < len; i += kChanThreads) one(i);
    if constexpr (sizeof(T) == 1) {
        // 32-bit sums of at most 1024 vectors (16384 * 255^2 < 2^32)
        for (long long i0 = tid; i0 < nv; i0 += 1024LL * kChanThreads) {
            uint32_t s1 = 0, s2 = 0;
            const long long i1 = min(nv, i0 + 1024LL * kChanThreads);
#pragma unroll 4
            for (long long i = i0; i < i1; i += kChanThreads) {
                const uint4 v = vec[i];
                s1 = __dp4a(v.x, 0x01010101u, s1);
                s1 = __dp4a(v.y, 0x01010101u, s1);
                s1 = __dp4a(v.z, 0x01010101u, s1);
                s1 = __dp4a(v.w, 0x01010101u, s1);
                s2 = __dp4a(v.x, v.x, s2);
                s2 = __dp4a(v.y, v.y, s2);
                s2 = __dp4a(v.z, v.z, s2);
                s2 = __dp4a(v.w, v.w, s2);
            }
            a1 += s1;
            a2 += s2;
        }
    } else {
        for (long long i0 = tid; i0 < nv; i0 += 1024LL * kChanThreads) {
            int s1 = 0;  // (8192 samples of at most 65535)
            const long long i1 = min(nv, i0 + 1024LL * kChanThreads);
#pragma unroll 4
            for (long long i = i0; i < i1; i += kChanThreads) {
                const uint4 v = vec[i];
                word_sums<T>(v.x, s1, a2);
                word_sums<T>(v.y, s1, a2);
                word_sums<T>(v.z, s1, a2);
                word_sums<T>(v.w, s1, a2);
            }
            a1 += s1;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        a2 += __shfl_xor_sync(0xffffffffu, a2, o);
    }
    __shared__ long long r1[kChanThreads / 32];
    __shared__ unsigned long long r2[kChanThreads / 32];
    __shared__ IntClip s_c;
    if ((tid & 31) == 0) {
        r1[tid >> 5] = a1;
        r2[tid >> 5] = a2;
    }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kChanThreads / 32; ++w) {
            a1 += r1[w];
            a2 += r2[w];
        }
        s_c = int_clip<T>(a1, (long long)a2, len, k);
    }
    __syncthreads();
    const IntClip c = s_c;
    auto clip_one = [&](long long i) {
        const int v = row[i];
        if (v <= c.lo || v >= c.hi) row[i] = (T)c.rep;
    };
    for (long long i = tid; i < head; i += kChanThreads) clip_one(i);
    for (long long i = tail + tid; i < len; i += kChanThreads) clip_one(i);
    WordClip<T> wc;
    const IntClip c4[4] = {c, c, c, c};
    wc.set(c4);
    // (the loads of a batch before its stores: a store orders the loads behind it)
    constexpr int U = 4;
    for (long long i0 = tid; i0 < nv; i0 += U * kChanThreads) {
        uint4 v[U];
#pragma unroll
        for (int j = 0; j < U; ++j)
            if (i0 + j * kChanThreads < nv) v[j] = vec[i0 + j * kChanThreads];
#pragma unroll
        for (int j = 0; j < U; ++j) {
            if (i0 + j * kChanThreads >= nv) break;
            const uint4 q = make_uint4(wc.apply(v[j].x), wc.apply(v[j].y), wc.apply(v[j].z),
                                       wc.apply(v[j].w));
            if (((q.x ^ v[j].x) | (q.y ^ v[j].y) | (q.z ^ v[j].z) | (q.w ^ v[j].w)) != 0u)
                vec[i0 + j * kChanThreads] = q;
        }
    }
}

constexpr int kSpecThreads = 512;  // 256 channels x 2 vectors of 16 bytes

// Spectra of integer samples: a cluster of CTAs takes 32 bytes of columns (32 uint8 spectra, 16
// of 16-bit samples) over all channels.  A thread holds the same 16-byte vector of NV channels
// in registers from the statistics to the clip, so the block is read once and only the vectors
// that change are written; the CTAs of the cluster (each 256 NV channels) add their columns'
// sums over distributed shared memory.  Past 8 x 2048 channels the threads take further batches
// of channels and read them again for the clip.  Rows start on 16-byte boundaries; columns at
// or past len are neither counted nor written.
template <typename T, int NV>
__global__ void __launch_bounds__(kSpecThreads, 2)
    k_clip_spectra_int(T *__restrict__ x, int nchans, long long stride, long long len, double k,
                       int nbatch)
{
    constexpr int SPW = 4 / (int)sizeof(T);  // samples per word
    constexpr int N = 4 * SPW;               // columns of a vector
    cg::cluster_group cl = cg::this_cluster();
    // (the wait comes before the first store to another CTA's memory, which may only be touched
    // once that CTA is known to run; the loads and sums between hide it)
    auto started = cl.barrier_arrive();
    const int rank = (int)cl.block_rank(), nrank = (int)cl.num_blocks();
    const int tid = threadIdx.x, half = tid & 1;
    const long long t0 = (long long)(blockIdx.x / nrank) * (2 * N) + half * N;
    const int ncol = (int)max(0LL, min((long long)N, len - t0));  // columns of this vector
    constexpr int NWARP = kSpecThreads / 32;
    __shared__ long long w1[NWARP][2 * N];              // each warp's column sums
    __shared__ unsigned long long w2[NWARP][2 * N];
    __shared__ long long sum1[8][2 * N];                // each CTA of the cluster's
    __shared__ unsigned long long sum2[8][2 * N];
    __shared__ IntClip clip[2 * N];
    const int warp = tid >> 5;

    uint32_t v[NV][4];
    auto channel = [&](int b, int i) {
        return ((b * nrank + rank) * NV + i) * (kSpecThreads / 2) + (tid >> 1);
    };
    auto load = [&](int b) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = channel(b, i);
            uint4 q = make_uint4(0u, 0u, 0u, 0u);  // (adds nothing)
            if (c < nchans) {
                const T *p = x + (size_t)c * (size_t)stride + t0;
                if (ncol == N) {
                    q = *reinterpret_cast<const uint4 *>(p);
                } else {
                    uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                    for (int e = 0; e < N; ++e)
                        if (e < ncol)
                            w[e / SPW] |= ((uint32_t)p[e] & (0xffffffffu >> (32 - 8 * sizeof(T))))
                                          << (8 * sizeof(T) * (e % SPW));
                    q = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            v[i][0] = q.x;
            v[i][1] = q.y;
            v[i][2] = q.z;
            v[i][3] = q.w;
        }
    };
    for (int b = 0; b < nbatch; ++b) {
        load(b);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            // the word's columns summed over this thread's channels, then over the 16 lanes of
            // the warp that hold the same columns
            if constexpr (sizeof(T) == 1) {
                uint32_t p01 = 0, p23 = 0, s2[4] = {0u, 0u, 0u, 0u};
                constexpr int G = (NV + 3) / 4;
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    // four channels' words as one word per column: dp4a adds the four samples
                    // (and their squares)
                    const uint32_t a = v[4 * g][w];
                    const uint32_t bb = 4 * g + 1 < NV ? v[(4 * g + 1) % NV][w] : 0u;
                    const uint32_t c = 4 * g + 2 < NV ? v[(4 * g + 2) % NV][w] : 0u;
                    const uint32_t d = 4 * g + 3 < NV ? v[(4 * g + 3) % NV][w] : 0u;
                    const uint32_t ab0 = __byte_perm(a, bb, 0x5140), ab2 = __byte_perm(a, bb, 0x7362);
                    const uint32_t cd0 = __byte_perm(c, d, 0x5140), cd2 = __byte_perm(c, d, 0x7362);
                    const uint32_t col[4] = {
                        __byte_perm(ab0, cd0, 0x5410), __byte_perm(ab0, cd0, 0x7632),
                        __byte_perm(ab2, cd2, 0x5410), __byte_perm(ab2, cd2, 0x7632)};
                    p01 = __dp4a(col[0], 0x01010101u, p01);
                    p01 += __dp4a(col[1], 0x01010101u, 0u) << 16;
                    p23 = __dp4a(col[2], 0x01010101u, p23);
                    p23 += __dp4a(col[3], 0x01010101u, 0u) << 16;
#pragma unroll
                    for (int e = 0; e < 4; ++e) s2[e] = __dp4a(col[e], col[e], s2[e]);
                }
                // (16-bit lanes: 16 lanes x NV channels x 255 < 2^16)
                static_assert(16 * NV * 255 < 65536, "packed column sums");
#pragma unroll
                for (int o = 16; o > 1; o >>= 1) {
                    p01 += __shfl_xor_sync(0xffffffffu, p01, o);
                    p23 += __shfl_xor_sync(0xffffffffu, p23, o);
#pragma unroll
                    for (int e = 0; e < 4; ++e) s2[e] += __shfl_xor_sync(0xffffffffu, s2[e], o);
                }
                if ((tid & 31) < 2) {
                    const uint32_t s1[4] = {p01 & 0xffffu, p01 >> 16, p23 & 0xffffu, p23 >> 16};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int q = half * N + 4 * w + e;
                        w1[warp][q] = (b ? w1[warp][q] : 0) + s1[e];
                        w2[warp][q] = (b ? w2[warp][q] : 0) + s2[e];
                    }
                }
            } else {
                int s1[2] = {0, 0};
                unsigned long long s2[2] = {0ull, 0ull};
#pragma unroll
                for (int i = 0; i < NV; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int u = word_sample<T>(v[i][w], e);
                        s1[e] += u;
                        s2[e] += (unsigned long long)((uint32_t)u * (uint32_t)u);
                    }
#pragma unroll
                for (int o = 16; o > 1; o >>= 1)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        s1[e] += __shfl_xor_sync(0xffffffffu, s1[e], o);
                        s2[e] += __shfl_xor_sync(0xffffffffu, s2[e], o);
                    }
                if ((tid & 31) < 2)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int q = half * N + 2 * w + e;
                        w1[warp][q] = (b ? w1[warp][q] : 0) + s1[e];
                        w2[warp][q] = (b ? w2[warp][q] : 0) + s2[e];
                    }
            }
        }
    }
    __syncthreads();
    cl.barrier_wait(std::move(started));
    if (tid < 2 * N) {
        long long s1 = 0;
        unsigned long long s2 = 0;
#pragma unroll
        for (int q = 0; q < NWARP; ++q) {
            s1 += w1[q][tid];
            s2 += w2[q][tid];
        }
        for (int r = 0; r < nrank; ++r) {  // to every CTA of the cluster
            *cl.map_shared_rank(&sum1[rank][tid], r) = s1;
            *cl.map_shared_rank(&sum2[rank][tid], r) = s2;
        }
    }
    cl.sync();  // every CTA's sums have arrived (no CTA touches another's memory after this)
    if (tid < 2 * N) {
        long long s1 = 0;
        unsigned long long s2 = 0;
        for (int r = 0; r < nrank; ++r) {
            s1 += sum1[r][tid];
            s2 += sum2[r][tid];
        }
        clip[tid] = int_clip<T>(s1, (long long)s2, nchans, k);
    }
    __syncthreads();
    for (int b = 0; b < nbatch; ++b) {
        if (nbatch > 1) load(b);
        uint32_t changed = 0;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            WordClip<T> wc;
            wc.set(&clip[half * N + SPW * w]);
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const uint32_t q = wc.apply(v[i][w]);
                changed |= (uint32_t)(q != v[i][w]) << i;
                v[i][w] = q;
            }
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = channel(b, i);
            if (!((changed >> i) & 1u) || c >= nchans) continue;
            T *p = x + (size_t)c * (size_t)stride + t0;
            if (ncol == N) {
                *reinterpret_cast<uint4 *>(p) = make_uint4(v[i][0], v[i][1], v[i][2], v[i][3]);
            } else {
#pragma unroll
                for (int e = 0; e < N; ++e)
                    if (e < ncol) p[e] = (T)word_sample<T>(v[i][e / SPW], e % SPW);
            }
        }
    }
}

// Spectra of integer samples whose rows do not start on 16-byte boundaries: one thread per time
// sample.
template <typename T>
__global__ void k_clip_spectra_any(T *__restrict__ x, int nchans, long long stride, long long len,
                                   double k)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= len) return;
    long long s1 = 0, s2 = 0;
    for (int c = 0; c < nchans; ++c) {
        const long long v = (long long)x[(size_t)c * stride + t];
        s1 += v;
        s2 += v * v;
    }
    const IntClip cb = int_clip<T>(s1, s2, nchans, k);
    for (int c = 0; c < nchans; ++c) {
        T *p = x + (size_t)c * stride + t;
        const int v = *p;
        if (v <= cb.lo || v >= cb.hi) *p = (T)cb.rep;
    }
}

// ------------------------------------------------------------------------------------------
// float samples
// ------------------------------------------------------------------------------------------
constexpr int kRun = 1024;  // samples of a left-to-right run

// p1 += v, p2 += v * v over consecutive samples (v * v is exact in double: one rounding each, as
// dmul + dadd).
template <bool kSum1, int U>
__device__ __forceinline__ void run_add(const float (&v)[U], double &p1, double &p2)
{
    uint32_t sp = 0;
#pragma unroll
    for (int j = 0; j < U; ++j) sp = max(sp, special_key(v[j]));
    if (sp < 0x7f000000u) {
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const double d = float_bits_double(__float_as_uint(v[j]));
            if (kSum1) p1 = __dadd_rn(p1, d);
            p2 = __fma_rn(d, d, p2);
        }
    } else {
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const double d = (double)v[j];
            if (kSum1) p1 = __dadd_rn(p1, d);
            p2 = __fma_rn(d, d, p2);
        }
    }
}

// Left-to-right double sums of n (at most 1024) samples and of their squares; ld(v, at) loads
// samples [at, at + 16), one(at) a single one.
template <class Ld, class One>
__device__ __forceinline__ double2 run_sums(int n, const Ld &ld, const One &one)
{
    constexpr int U = 16;
    double p1 = 0.0, p2 = 0.0;
    CutSum cs;
    float a[U], b[U];
    const int n2 = n / (2 * U) * (2 * U);
    float big = 0.0f;
    if (n2) {
        ld(a, 0);
        // maxima of four samples, two by two the smaller, of these the larger: outliers among the
        // first samples do not move it
        float m[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            m[j] = fmaxf(fmaxf(fabsf(a[4 * j]), fabsf(a[4 * j + 1])),
                         fmaxf(fabsf(a[4 * j + 2]), fabsf(a[4 * j + 3])));
        big = fmaxf(fminf(m[0], m[1]), fminf(m[2], m[3]));
    }
    cs.start(big);
    for (int i = 0; i < n2; i += 2 * U) {  // the next 16 samples are loaded before these are added
        ld(b, i + U);
        cs.add(a);
        run_add<false, U>(a, p1, p2);
        if (i + 2 * U < n2) ld(a, i + 2 * U);
        cs.add(b);
        run_add<false, U>(b, p1, p2);
    }
    for (int i = n2; i < n; ++i) {
        const float v[1] = {one(i)};
        cs.add(v);
        run_add<false, 1>(v, p1, p2);
    }
    if (cs.ok()) return make_double2(cs.sum(), p2);
    for (int i = 0; i < n2; i += U) {
        ld(a, i);
#pragma unroll
        for (int j = 0; j < U; ++j)
            p1 = __dadd_rn(p1, special_key(a[j]) < 0x7f000000u
                                   ? float_bits_double(__float_as_uint(a[j]))
                                   : (double)a[j]);
    }
    for (int i = n2; i < n; ++i) p1 = __dadd_rn(p1, (double)one(i));
    return make_double2(p1, p2);
}

struct FloatClip {
    float lo, hi, rep;
};

__device__ __forceinline__ FloatClip float_clip(double s1, double s2, double n, double k)
{
    const double mu = __ddiv_rn(s1, n);
    const double var = __dadd_rn(__ddiv_rn(s2, n), -__dmul_rn(mu, mu));
    const double sig = var > 0.0 ? __dsqrt_rn(var) : 0.0;
    FloatClip c;
    clip_bounds_f32(mu, __dmul_rn(k, sig), &c.lo, &c.hi);
    c.rep = __double2float_rn(mu);
    return c;
}

constexpr int kChanF32Threads = 256;
constexpr int kChanF32Runs = 128;  // runs of a CTA's rows that the row count aims at

// Channels of float samples: a CTA takes `rpc` rows, one thread per run of 1024 samples of a
// row (left to right), then the runs' sums left to right, then the clip in float.  Several rows
// a CTA because a warp of double operations costs the same with few lanes as with 32.
__global__ void __launch_bounds__(kChanF32Threads, 3)
    k_clip_channels_f32(float *__restrict__ x, int nchans, long long stride, long long len,
                        double k, int rpc)
{
    extern __shared__ __align__(16) unsigned char sm[];
    double2 *part = reinterpret_cast<double2 *>(sm);  // [rpc][nruns]
    __shared__ FloatClip clip[kChanF32Runs];
    const int tid = threadIdx.x;
    const int c0 = blockIdx.x * rpc, rows = min(rpc, nchans - c0);
    const int nruns = (int)((len + kRun - 1) / kRun);
    const bool vec = (((uintptr_t)x | (uintptr_t)(stride * 4)) & 15) == 0;
    for (int q = tid; q < rows * nruns; q += kChanF32Threads) {
        const int r = q / nruns;
        const long long i0 = (long long)(q - r * nruns) * kRun;
        const float *p = x + (size_t)(c0 + r) * (size_t)stride + i0;
        const int n = (int)min((long long)kRun, len - i0);
        auto one = [&](int i) { return p[i]; };
        if (vec)
            part[q] = run_sums(
                n,
                [&](float (&d)[16], int at) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 u = *reinterpret_cast<const float4 *>(p + at + 4 * j);
                        d[4 * j] = u.x;
                        d[4 * j + 1] = u.y;
                        d[4 * j + 2] = u.z;
                        d[4 * j + 3] = u.w;
                    }
                },
                one);
        else
            part[q] = run_sums(
                n,
                [&](float (&d)[16], int at) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) d[j] = p[at + j];
                },
                one);
    }
    __syncthreads();
    for (int r = tid; r < rows; r += kChanF32Threads) {
        double s1 = 0.0, s2 = 0.0;
        for (int j = 0; j < nruns; ++j) {
            const double2 d = part[r * nruns + j];
            s1 = __dadd_rn(s1, d.x);
            s2 = __dadd_rn(s2, d.y);
        }
        clip[r] = float_clip(s1, s2, (double)len, k);
    }
    __syncthreads();
    for (int r = 0; r < rows; ++r) {
        float *row = x + (size_t)(c0 + r) * (size_t)stride;
        const FloatClip c = clip[r];
        auto bad = [&](float v) { return v <= c.lo || v >= c.hi; };
        long long done = 0;
        if (vec) {
            const long long nv = len / 4;
            done = nv * 4;
            // (the loads of a batch before its stores: a store orders the loads behind it)
            constexpr int U = 4;
            float4 *rv = reinterpret_cast<float4 *>(row);
            for (long long i0 = tid; i0 < nv; i0 += U * kChanF32Threads) {
                float4 v[U];
#pragma unroll
                for (int j = 0; j < U; ++j)
                    if (i0 + j * kChanF32Threads < nv) v[j] = rv[i0 + j * kChanF32Threads];
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    if (i0 + j * kChanF32Threads >= nv) break;
                    float4 &q = v[j];
                    if (bad(q.x) || bad(q.y) || bad(q.z) || bad(q.w)) {
                        q.x = bad(q.x) ? c.rep : q.x;
                        q.y = bad(q.y) ? c.rep : q.y;
                        q.z = bad(q.z) ? c.rep : q.z;
                        q.w = bad(q.w) ? c.rep : q.w;
                        rv[i0 + j * kChanF32Threads] = q;
                    }
                }
            }
        }
        for (long long i = done + tid; i < len; i += kChanF32Threads)
            if (bad(row[i])) row[i] = c.rep;
    }
}

constexpr int kSpecF32Threads = 256;

// Spectra of float samples: COLS columns a CTA, kSpecF32Threads / COLS threads a column; a thread
// sums runs of 1024 channels of its column left to right, one thread a column adds the runs left
// to right, then all threads clip.  128 columns where that leaves two CTAs a SM: the four warps
// that sum then lie on the SM's four schedulers, each with its own double unit; 32 columns
// otherwise.
template <int COLS>
__global__ void __launch_bounds__(kSpecF32Threads)
    k_clip_spectra_f32(float *__restrict__ x, int nchans, long long stride, long long len, double k)
{
    constexpr int kRows = kSpecF32Threads / COLS;
    __shared__ double2 part[kRows][COLS];
    __shared__ FloatClip clip[COLS];
    const int lane = threadIdx.x, ty = threadIdx.y;
    const long long t = (long long)blockIdx.x * COLS + lane;
    const bool in = t < len;
    const int nruns = (nchans + kRun - 1) / kRun;
    double s1 = 0.0, s2 = 0.0;  // (threads ty 0)
    for (int r0 = 0; r0 < nruns; r0 += kRows) {
        const int r = r0 + ty;
        const int ca = r * kRun, cb = min(ca + kRun, nchans);
        double2 sums = make_double2(0.0, 0.0);
        if (in && r < nruns) {
            const float *p = x + (size_t)ca * (size_t)stride + t;
            sums = run_sums(
                cb - ca,
                [&](float (&d)[16], int at) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) d[j] = p[(size_t)(at + j) * (size_t)stride];
                },
                [&](int i) { return p[(size_t)i * (size_t)stride]; });
        }
        if (r0 > 0) __syncthreads();  // the previous runs are added
        part[ty][lane] = sums;
        __syncthreads();
        if (ty == 0)
            for (int j = 0; j < min(kRows, nruns - r0); ++j) {
                s1 = __dadd_rn(s1, part[j][lane].x);
                s2 = __dadd_rn(s2, part[j][lane].y);
            }
    }
    if (ty == 0 && in) clip[lane] = float_clip(s1, s2, (double)nchans, k);
    __syncthreads();
    if (!in) return;
    const FloatClip c = clip[lane];
    constexpr int U = 16;
    for (int ch = ty; ch < nchans; ch += U * kRows) {
        float *p = x + (size_t)ch * (size_t)stride + t;
        const size_t step = (size_t)kRows * (size_t)stride;
        float v[U];
#pragma unroll
        for (int j = 0; j < U; ++j) v[j] = ch + j * kRows < nchans ? p[j * step] : c.rep;
#pragma unroll
        for (int j = 0; j < U; ++j)
            if (ch + j * kRows < nchans && (v[j] <= c.lo || v[j] >= c.hi)) p[j * step] = c.rep;
    }
}

// ------------------------------------------------------------------------------------------
// launches
// ------------------------------------------------------------------------------------------
template <typename T, int NV>
mdsm_status launch_spectra_int(T *x, int nchans, long long stride, long long len, double ks,
                               cudaStream_t st)
{
    constexpr int N = 16 / (int)sizeof(T);
    const int per = kSpecThreads / 2 * NV;
    const int ncl = std::min(8, (nchans + per - 1) / per);
    const int nbatch = (nchans + per * ncl - 1) / (per * ncl);
    const long long tiles = (len + 2 * N - 1) / (2 * N);
    if (tiles * ncl > 0x7fffffffLL) return fail(MDSM_EINVAL, "rfi clip: block too long");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * ncl));
    cfg.blockDim = dim3(kSpecThreads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ncl;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    MDSM_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_clip_spectra_int<T, NV>, x, nchans, stride, len, ks,
                                     nbatch));
    return MDSM_OK;
}

template <typename T>
mdsm_status clip_int(T *x, int nchans, long long stride, long long len, double kc, double ks,
                     cudaStream_t st)
{
    if (kc > 0.0) {
        k_clip_channels_int<T><<<nchans, kChanThreads, 0, st>>>(x, stride, len, kc);
        MDSM_CUDA_TRY(cudaGetLastError());
    }
    if (ks > 0.0) {
        // the vector form where every row starts on a 16-byte boundary; few channels take two
        // vectors a thread (512 channels a CTA) instead of eight
        if ((((uintptr_t)x | (uintptr_t)(stride * (long long)sizeof(T))) & 15) == 0)
            return nchans <= kSpecThreads ? launch_spectra_int<T, 2>(x, nchans, stride, len, ks, st)
                                          : launch_spectra_int<T, 8>(x, nchans, stride, len, ks, st);
        k_clip_spectra_any<T><<<(unsigned)((len + 255) / 256), 256, 0, st>>>(x, nchans, stride, len,
                                                                             ks);
        MDSM_CUDA_TRY(cudaGetLastError());
    }
    return MDSM_OK;
}

mdsm_status clip_f32(float *x, int nchans, long long stride, long long len, double kc, double ks,
                     cudaStream_t st)
{
    if (kc > 0.0) {
        const long long nruns = (len + kRun - 1) / kRun;
        if (nruns * (long long)sizeof(double2) > 200 * 1024)
            return fail(MDSM_EINVAL, "rfi clip: row too long");
        // rows a CTA: enough runs for its threads, while two CTAs a SM remain
        const int rpc = (int)std::max<long long>(
            1, std::min<long long>({kChanF32Runs / nruns, (nchans + 303) / 304}));
        // (close to a third of a SM's shared memory: at most three CTAs share its double units)
        const size_t smem = std::max<size_t>((size_t)(rpc * nruns) * sizeof(double2), 72 * 1024);
        MDSM_CUDA_TRY(cudaFuncSetAttribute(k_clip_channels_f32,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_clip_channels_f32<<<(nchans + rpc - 1) / rpc, kChanF32Threads, smem, st>>>(
            x, nchans, stride, len, kc, rpc);
        MDSM_CUDA_TRY(cudaGetLastError());
    }
    if (ks > 0.0) {
        if (len >= 304 * 128)
            k_clip_spectra_f32<128>
                <<<(unsigned)((len + 127) / 128), dim3(128, kSpecF32Threads / 128), 0, st>>>(
                    x, nchans, stride, len, ks);
        else
            k_clip_spectra_f32<32>
                <<<(unsigned)((len + 31) / 32), dim3(32, kSpecF32Threads / 32), 0, st>>>(
                    x, nchans, stride, len, ks);
        MDSM_CUDA_TRY(cudaGetLastError());
    }
    return MDSM_OK;
}

}  // namespace

mdsm_status rfi_clip(void *d_x, int dtype, int nchans, long long stride, long long len,
                     double k_chan, double k_spec, cudaStream_t st)
{
    switch (dtype) {
    case MDSM_U8:
        return clip_int(static_cast<uint8_t *>(d_x), nchans, stride, len, k_chan, k_spec, st);
    case MDSM_U16:
        return clip_int(static_cast<uint16_t *>(d_x), nchans, stride, len, k_chan, k_spec, st);
    case MDSM_I16:
        return clip_int(static_cast<int16_t *>(d_x), nchans, stride, len, k_chan, k_spec, st);
    case MDSM_F32:
        return clip_f32(static_cast<float *>(d_x), nchans, stride, len, k_chan, k_spec, st);
    }
    return fail(MDSM_EINVAL, "rfi clip: unknown sample type");
}

}  // namespace mdsm
