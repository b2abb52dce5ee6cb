// groupsum.cu -- brute-force dedispersion of 8- and 16-bit samples by sums of groups of channels: the exact
// integer sums of dedisp.cu's packed kernels with fewer additions.
//
// Across a block of neighbouring DM trials the shifts of a few neighbouring channels, taken relative to the
// first one's, follow only a few patterns (4096 channels of 300 MHz: 8 channels have 7-9 patterns in 60
// trials).  So each pattern is summed once, into shared memory, and a trial adds one word of its pattern
// per group where the packed kernels add one per channel.  Integer sums do not depend on their order.
//
// One CTA: NW warps of DPW trials each x 512 samples, and a warp that copies.  The channels come in chunks
// of a few groups: rows by bulk copies, three chunks ahead (16-bit samples two), with the chunk's tables.
// The compute warps take tasks (a segment of a run of patterns): the run's first pattern adds the group's
// rows, each further one swaps the rows in which it differs (gs_patterns).  Then each adds the patterns for
// its trials (gs_add).  A warp works on chunk k + 1's tasks before it adds chunk k, over three pattern
// buffers, so warps without a task, or with a longer one, do not hold the others up at a barrier.
//
// Groups of 8, 4, 2 or 1 channels are chosen where the tables are made, by the wavefronts that they take:
// 8 where a block's trials share patterns well (4096 channels, steps of 0.24 pc cm^-3), 4 and less where
// channels are wide or steps coarse.
//
// What bounds it: instruction issue (69 %), then shared memory (59 %): a pattern costs about 45 instructions
// and 9 wavefronts a step, an add 2 and 1 a word.  4096 channels x 2^18 samples x 4096 trials: 206 ms by the
// packed kernel (which is near its own bounds: 80 % shared memory, 70 % integer pipe), 132 ms here.  2048
// channels of 16-bit samples x 30011 x 517: 3.09 -> 2.14 ms.  With one barrier a chunk and two buffers it
// took 188 ms; tasks of whole groups 206 (too few warps with a task); one word a lane and task 198 (decoding);
// 19 warps of 3 trials 147, 11 of 6 135, five words a lane 154, four smaller buffers 146.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <new>
#include <thread>
#include <type_traits>
#include <utility>
#include <vector>

#include "internal.h"
#include "ptx.cuh"

namespace mdsm {

namespace {

constexpr int kGsT = 512;           // samples of a tile
// Stages of rows: uint8 three (short parts want the copies' lead), 16-bit samples two half as large again
// (their wider rows would leave chunks of one group; 2048 channels 2.29 -> 2.13 ms).
__host__ __device__ constexpr int gs_raw(int sw) { return sw == 1 ? 3 : 2; }
__host__ __device__ constexpr int gs_rawcap(int sw) { return 42 * 1024 / gs_raw(sw); }
constexpr int kGsBlobs = 5;         // entries of tables: a chunk's are read until its sums are added
constexpr int kGsZ = 3;             // pattern buffers
constexpr int kGsRows = 32;         // channels of a chunk, at most
constexpr int kGsGroups = 16;       // groups of a chunk, at most
constexpr int kGsG = 8;             // channels of a group, at most
constexpr int kGsTasks = 127;       // tasks of a chunk, at most
constexpr int kGsRunMin = 3;        // patterns of a run, at least (where the group has them)
constexpr int kGsTurn = 7;          // warps by which a chunk's first task moves
constexpr int kGsPad = 16;          // bytes before a staged row (a pattern may start below its smin)
constexpr int kGsHead = 256;        // barriers and chunk headers
constexpr int kGsLast = 1, kGsStop = 2;  // chunk flags
constexpr uint32_t kGsNone = 0xffffffffu;  // a step that stores no pattern
constexpr int kGsU = 3;             // words of a row that a lane adds: 3 words apart, lanes do not conflict

// A task is one segment of a group's patterns: 32 lanes of kGsU words; uint8 lanes need the next one's
// first sample, so the last lane stores nothing and segments are 31 lanes apart.
__host__ __device__ constexpr int gs_lanes(int sw) { return sw == 1 ? 31 : 32; }
// Samples that a segment covers, and the words of a pattern's row where the widest span of a chunk's
// groups is `span`, to whole lanes: uint8, pairs of 16-bit sums from an even and (again as many words) from
// an odd sample on; 16-bit samples, 32-bit sums.
__host__ __device__ constexpr int gs_seg(int sw) { return gs_lanes(sw) * kGsU * 4 / sw; }
__host__ __device__ constexpr int gs_row_words(int sw, int span)
{
    return sw == 1 ? 2 * 2 * kGsU * ((kGsT + span + 4 * kGsU) / (4 * kGsU))
                   : 2 * kGsU * ((kGsT + span + 2 * kGsU - 1) / (2 * kGsU));
}

}  // namespace

struct GsArgs {
    const unsigned char *in;
    long long in_stride;    // elements
    unsigned char *out;
    long long out_stride;   // elements
    const uint4 *blobs;     // the chunks' tables
    const int4 *chunks;     // tables' first entry, their bytes, first channel, and in bits: channels,
                            // groups << 6, tasks << 16, 16-byte units of a staged row << 23
    const int *chunk0;      // [nblk + 1] first chunk of a DM block
    const int2 *chan;       // [blk][c] smallest shift, span
    int nchans, ndms, nsamp, nblk, ntiles, nitems, nsplit;
    int rawcap, blobcap, zcap;  // bytes of a stage, of a tables' entry; words of a pattern buffer
    int out_i32;
    unsigned *err;
    unsigned long long *mom;
};

namespace {

// A word's lower (0) or upper (1) 16 bits widened to 32.
template <bool SIGNED, int HI>
__device__ __forceinline__ uint32_t gs_half(uint32_t w)
{
    if constexpr (HI)
        return SIGNED ? (uint32_t)((int32_t)w >> 16) : w >> 16;
    else
        return SIGNED ? (uint32_t)(int32_t)(int16_t)w : w & 0xffffu;
}

// One segment of a group's patterns, each the sum of the group's rows at the pattern's offsets.  The first
// pattern adds the rows, two a step; each further one swaps, a step each, the rows in which it differs
// from the one before (its offset's words added, the old ones' taken off).
// Step: two rows' first words (bytes), their shifts (bits 0-4 and 8-12; bit 16: the first row only), the
// first word of the pattern that the sum is by now, or kGsNone.
template <int SW, bool SIGNED>
__device__ __forceinline__ void gs_patterns(const uint4 *steps, int nsteps, int nfirst,
                                            const unsigned char *rows, uint32_t *z, int seg, int lane,
                                            int zcopy)
{
    constexpr int U = kGsU;
    const int at = (seg * gs_lanes(SW) + lane) * U;
    const unsigned char *base = rows + at * 4;
    uint32_t *zb = z + at * 2;
    const bool mine = at * 2 < zcopy && (SW == 2 || lane < 31);
    uint32_t A[U] = {}, O[U] = {};  // uint8: raw words and their odd samples (mod 2^32, exact again at
                                    // every stored pattern); 16-bit samples: the two samples' sums
    uint32_t wx[U + 1], wy[U + 1];
    auto load = [&](const uint4 &st) {
        const uint32_t *px = reinterpret_cast<const uint32_t *>(base + st.x);
        const uint32_t *py = reinterpret_cast<const uint32_t *>(base + st.y);
#pragma unroll
        for (int u = 0; u <= U; ++u) {
            wx[u] = px[u];
            wy[u] = py[u];
        }
    };
    auto shifted = [&](uint32_t z, uint32_t (&x)[U], uint32_t (&y)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            x[u] = __funnelshift_r(wx[u], wx[u + 1], z);
            y[u] = __funnelshift_r(wy[u], wy[u + 1], z >> 8);
        }
    };
    auto store = [&](uint32_t word) {
        uint2 *p = reinterpret_cast<uint2 *>(zb + word);
        if constexpr (SW == 1) {
            uint32_t E[U + 1];  // samples 0 and 2 of a word; O: 1 and 3
#pragma unroll
            for (int u = 0; u < U; ++u) E[u] = A[u] - (O[u] << 8);
            E[U] = __shfl_down_sync(0xffffffffu, E[0], 1);
            if (mine) {
                uint2 *p1 = reinterpret_cast<uint2 *>(zb + word + zcopy);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    p[u] = make_uint2(__byte_perm(E[u], O[u], 0x5410), __byte_perm(E[u], O[u], 0x7632));
                    p1[u] = make_uint2(__byte_perm(O[u], E[u], 0x7610),
                                       __byte_perm(O[u], E[u + 1], 0x5432));
                }
            }
        } else if (mine) {
#pragma unroll
            for (int u = 0; u < U; ++u) p[u] = make_uint2(A[u], O[u]);
        }
    };
    // the next step's words are on their way while one is added (the entry after the last step is
    // another run's or an offset's: read as a step of the first row, and not used)
    uint4 cur = steps[0];
    load(cur);
    uint4 next = steps[1];
#pragma unroll 1
    for (int i = 1;; ++i) {
        uint32_t x[U], y[U];
        shifted(cur.z, x, y);
        const uint32_t one = cur.z >> 16, word = cur.w;
        cur = next;
        if (i >= nsteps) cur.x = cur.y = 0u;
        load(cur);
        next = steps[i + 1];
        if (one)
#pragma unroll
            for (int u = 0; u < U; ++u) y[u] = 0u;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if constexpr (SW == 1) {
                A[u] += x[u] + y[u];
                O[u] += __byte_perm(x[u], 0u, 0x4341) + __byte_perm(y[u], 0u, 0x4341);
            } else {
                A[u] += gs_half<SIGNED, 0>(x[u]) + gs_half<SIGNED, 0>(y[u]);
                O[u] += gs_half<SIGNED, 1>(x[u]) + gs_half<SIGNED, 1>(y[u]);
            }
        }
        if (word != kGsNone) {
            store(word);
            break;
        }
    }
#pragma unroll 1
    for (int i = nfirst + 1; i <= nsteps; ++i) {
        uint32_t x[U], y[U];
        shifted(cur.z, x, y);
        const uint32_t word = cur.w;
        cur = next;
        if (i >= nsteps) cur.x = cur.y = 0u;
        load(cur);
        next = steps[i + 1];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if constexpr (SW == 1) {
                A[u] += x[u] - y[u];
                O[u] += __byte_perm(x[u], 0u, 0x4341) - __byte_perm(y[u], 0u, 0x4341);
            } else {
                A[u] += gs_half<SIGNED, 0>(x[u]) - gs_half<SIGNED, 0>(y[u]);
                O[u] += gs_half<SIGNED, 1>(x[u]) - gs_half<SIGNED, 1>(y[u]);
            }
        }
        if (word != kGsNone) store(word);
    }
}

// Offsets of a warp in a group's tables (its trials', to a power of two), and of the group (whole
// 16-byte units).
__host__ __device__ constexpr int gs_entry(int dpw) { return dpw > 4 ? 8 : 4; }
__host__ __device__ constexpr int gs_offsets(int nw, int dpw) { return (nw * gs_entry(dpw) + 7) / 8 * 8; }

template <int SW, int DPW>
struct GsAcc {
    static constexpr int NR = SW == 1 ? kGsT / 64 : kGsT / 32;  // words a lane reads of a trial
    static constexpr int NO = SW == 1 ? NR : 1;
    uint32_t a[DPW][NR];  // uint8: pairs summed mod 2^32; 16-bit samples: the sums
    uint32_t o[DPW][NO];  // uint8: the odd samples' sums
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int j = 0; j < DPW; ++j) {
#pragma unroll
            for (int r = 0; r < NR; ++r) a[j][r] = 0u;
#pragma unroll
            for (int r = 0; r < NO; ++r) o[j][r] = 0u;
        }
    }
};

// o + (w >> 16), on the multiply-add pipe.
__device__ __forceinline__ uint32_t gs_add_hi(uint32_t w, uint32_t o)
{
    uint32_t d;
    asm("mad.hi.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(w), "r"(0x10000u), "r"(o));
    return d;
}

// The groups' patterns added for the warp's trials, up to four groups a step (uint8: their sums stay
// within the 16-bit halves, so the odd samples' are taken once).  offs: the warp's of the first group.
template <int SW, int DPW, int NW>
__device__ __forceinline__ void gs_add(GsAcc<SW, DPW> &acc, const uint32_t *z, const uint16_t *offs,
                                       int ng)
{
    constexpr int NR = GsAcc<SW, DPW>::NR, NB = 8;  // words at a time
    using Entry = std::conditional_t<gs_entry(DPW) == 8, uint4, uint2>;
    auto step = [&](auto count, int g) {
        constexpr int N = decltype(count)::value;
        union {
            Entry e;
            uint32_t w[gs_entry(DPW) / 2];
        } v[N];
#pragma unroll
        for (int n = 0; n < N; ++n)
            v[n].e = *reinterpret_cast<const Entry *>(offs + (g + n) * gs_offsets(NW, DPW));
#pragma unroll
        for (int j = 0; j < DPW; ++j) {
            const uint32_t *p[N];
#pragma unroll
            for (int n = 0; n < N; ++n)
                p[n] = z + (j & 1 ? v[n].w[j / 2] >> 16 : v[n].w[j / 2] & 0xffffu);
#pragma unroll
            for (int r0 = 0; r0 < NR; r0 += NB) {
                uint32_t w[N][NB];
#pragma unroll
                for (int r = 0; r < NB; ++r)
#pragma unroll
                    for (int n = 0; n < N; ++n) w[n][r] = p[n][32 * (r0 + r)];
#pragma unroll
                for (int r = 0; r < NB; ++r) {
                    uint32_t t = w[0][r];
                    if constexpr (N == 2) t += w[1][r];
                    if constexpr (N > 2) t += w[1][r] + w[2][r];
                    if constexpr (N > 3) t += w[3][r];
                    acc.a[j][r0 + r] += t;
                    if constexpr (SW == 1) acc.o[j][r0 + r] = gs_add_hi(t, acc.o[j][r0 + r]);
                }
            }
        }
    };
    int g = 0;
#pragma unroll 1
    for (; g + 4 <= ng; g += 4) step(std::integral_constant<int, 4>(), g);
    if (ng - g == 3) step(std::integral_constant<int, 3>(), g);
    if (ng - g == 2) step(std::integral_constant<int, 2>(), g);
    if (ng - g == 1) step(std::integral_constant<int, 1>(), g);
}

// Stores a trial's sums (and folds its moments).
template <int SW, int DPW, int NW>
__device__ __forceinline__ void gs_store(const GsArgs &a, const GsAcc<SW, DPW> &acc, int blk, int tile,
                                         int warp, int lane)
{
    constexpr int NR = GsAcc<SW, DPW>::NR, SPW = SW == 1 ? 2 : 1;
    const long long t0 = (long long)tile * kGsT;
#pragma unroll
    for (int j = 0; j < DPW; ++j) {
        const int d = (blk * NW + warp) * DPW + j;
        if (d >= a.ndms) continue;  // (the whole warp)
        unsigned char *orow = a.out + (size_t)((long long)d * a.out_stride) * 4;
        long long m1 = 0;
        unsigned long long m2lo = 0, m2hi = 0;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const long long t = t0 + SPW * (lane + 32 * r);
            int32_t v[SPW];
            if constexpr (SW == 1) {
                v[0] = (int32_t)(acc.a[j][r] - (acc.o[j][r] << 16));
                v[SPW - 1] = (int32_t)acc.o[j][r];
            } else {
                v[0] = (int32_t)acc.a[j][r];
            }
            if (a.mom) {
#pragma unroll
                for (int e = 0; e < SPW; ++e)
                    if (t + e < a.nsamp) {
                        const unsigned long long q =
                            (unsigned long long)((long long)v[e] * (long long)v[e]);
                        m1 += v[e];
                        m2lo += q;
                        m2hi += (m2lo < q);
                    }
            }
            if (a.nsplit > 1) {  // a part of the channels adds its sums
#pragma unroll
                for (int e = 0; e < SPW; ++e)
                    if (t + e < a.nsamp) {
                        if (a.out_i32)
                            atomicAdd(reinterpret_cast<int *>(orow) + t + e, v[e]);
                        else  // (whole numbers below 2^24: exact in any order)
                            atomicAdd(reinterpret_cast<float *>(orow) + t + e, (float)v[e]);
                    }
                continue;
            }
            if (SPW == 2 && t + 1 < a.nsamp && ((uintptr_t)(orow + t * 4) & 7) == 0) {
                if (a.out_i32)
                    *reinterpret_cast<int2 *>(orow + t * 4) = make_int2(v[0], v[SPW - 1]);
                else
                    *reinterpret_cast<float2 *>(orow + t * 4) =
                        make_float2((float)v[0], (float)v[SPW - 1]);
            } else {
#pragma unroll
                for (int e = 0; e < SPW; ++e)
                    if (t + e < a.nsamp) {
                        if (a.out_i32)
                            reinterpret_cast<int *>(orow)[t + e] = v[e];
                        else
                            reinterpret_cast<float *>(orow)[t + e] = (float)v[e];
                    }
            }
        }
        if (a.mom) {
            // the row's share of this item: warp sum (128-bit with carries), then one atomic per
            // word; integer sums do not depend on their order
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                m1 += __shfl_xor_sync(0xffffffffu, m1, o);
                const unsigned long long lo = __shfl_xor_sync(0xffffffffu, m2lo, o);
                const unsigned long long hi = __shfl_xor_sync(0xffffffffu, m2hi, o);
                const unsigned long long nl = m2lo + lo;
                m2hi += hi + (nl < m2lo);
                m2lo = nl;
            }
            if (lane == 0) {
                unsigned long long *mp = a.mom + 3 * (size_t)d;
                atomicAdd(mp, (unsigned long long)m1);
                const unsigned long long old = atomicAdd(mp + 1, m2lo);
                atomicAdd(mp + 2, m2hi + (old + m2lo < old ? 1ull : 0ull));
            }
        }
    }
}

// True in every lane, or (a lane's wait ran out) false in every lane.
__device__ __forceinline__ bool gs_wait(uint64_t *bar, uint32_t parity, unsigned *err)
{
    return !__any_sync(0xffffffffu, !mbar_wait_bounded(bar, parity, err, ERR_WAIT_TIMEOUT));
}

// NW compute warps of DPW trials each, and a warp that copies.  15 x 4 trials (128 registers a thread) where
// the trials fill its blocks, 19 x 2 (96) for few trials or short calls.
template <int SW, int NW, int DPW, bool SIGNED>
__global__ void __launch_bounds__((NW + 1) * 32, 1) k_group_sum(const __grid_constant__ GsArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int RAW = gs_raw(SW);
    // a chunk's copies have landed / its patterns are stored (and its rows free) / its sums are added
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *built = full + RAW, *added = built + kGsZ;
    int4 *meta = reinterpret_cast<int4 *>(smem + 96);  // kGsBlobs: item, chunk bits, table bytes, flags
    unsigned char *blobs = smem + kGsHead;
    uint32_t *Z = reinterpret_cast<uint32_t *>(blobs + kGsBlobs * a.blobcap);
    unsigned char *raw = reinterpret_cast<unsigned char *>(Z + kGsZ * a.zcap);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < RAW; ++s) mbar_init(&full[s], 1);
        for (int s = 0; s < kGsZ; ++s) {
            mbar_init(&built[s], NW);
            mbar_init(&added[s], NW);
        }
        fence_mbar_init();
    }
    __syncthreads();

    // item: DM block fastest (from tile to tile a different one first, so that a CTA does not meet the
    // same block, perhaps the costliest, in each of its items), then the time tile, then the part of the
    // channels
    auto chunks_of = [&](int it, int &blk, int &tile) {
        const int rest = it / a.nblk;
        blk = (int)(((unsigned)it + (unsigned)rest) % (unsigned)a.nblk);
        tile = rest % a.ntiles;
        const int part = rest / a.ntiles;
        const int k0 = __ldg(a.chunk0 + blk), n = __ldg(a.chunk0 + blk + 1) - k0;
        return make_int2(k0 + (int)((long long)n * part / a.nsplit),
                         k0 + (int)((long long)n * (part + 1) / a.nsplit));
    };

    if (warp == NW) {
        // ---- the copies, RAW chunks ahead, across items ----
        int it = (int)blockIdx.x - (int)gridDim.x, blk = 0, tile = 0, k = 0;
        int2 ks = make_int2(0, 0);
        int4 ck = make_int4(0, 0, 0, 0);
        int2 ch = make_int2(0, 0);
        bool done = false;
        auto load = [&]() {  // the next chunk's entries, a fill ahead
            while (!done && k >= ks.y) {  // (a part may have no chunk: then its item has no store)
                it += gridDim.x;
                done = it >= a.nitems;
                if (!done) {
                    ks = chunks_of(it, blk, tile);
                    k = ks.x;
                }
            }
            if (done) return;
            ck = __ldg(a.chunks + k);
            if (lane < (ck.w & 63)) ch = __ldg(a.chan + (size_t)blk * a.nchans + ck.z + lane);
        };
        load();
        auto fill = [&](unsigned n) {  // chunk n of the stream
            const int s = (int)(n % RAW), e = (int)(n % kGsBlobs);
            if (done) {
                if (lane == 0) {
                    meta[e] = make_int4(-1, 0, 0, kGsStop);
                    mbar_arrive(&full[s]);
                }
                __syncwarp();
                return;
            }
            const int rows = ck.w & 63, pitch = (ck.w >> 23) * 16;
            const long long t0 = (long long)tile * kGsT;
            unsigned bytes = 0;
            const unsigned char *src = nullptr;
            if (lane < rows) {
                const long long start = t0 + ch.x;
                // (no sample past the last output's is read)
                const long long end = start + min((long long)kGsT, (long long)a.nsamp - t0) + ch.y;
                const long long sb = (start * SW) & ~15LL, eb = (end * SW + 15) & ~15LL;
                bytes = (unsigned)(eb - sb);
                src = a.in + (size_t)(ck.z + lane) * (size_t)a.in_stride * SW + sb;
            }
            unsigned total = bytes;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
            __syncwarp();
            if (lane == 0) {
                meta[e] = make_int4(it, ck.w, ck.y, k == ks.y - 1 ? kGsLast : 0);
                mbar_arrive_expect_tx(&full[s], total + (unsigned)ck.y);
            }
            __syncwarp();
            if (lane < rows)
                bulk_g2s(raw + s * a.rawcap + lane * pitch + kGsPad, src, bytes, &full[s]);
            if (lane == 0)
                bulk_g2s(blobs + e * a.blobcap, a.blobs + ck.x, (unsigned)ck.y, &full[s]);
            ++k;
            load();
        };
        for (unsigned n = 0; n < RAW; ++n) fill(n);
        for (unsigned k2 = 0;; ++k2) {
            if ((meta[k2 % kGsBlobs].w & kGsStop) != 0) return;  // (written by this warp)
            // chunk k2's rows are free, and the tables of chunk k2 - 2 (its sums were added before any
            // warp began with chunk k2's patterns)
            if (!gs_wait(&built[k2 % kGsZ], (k2 / kGsZ) & 1u, a.err)) {
                // let the copies already issued land before the CTA exits (bounded as well)
                for (unsigned q = k2; q < k2 + RAW; ++q)
                    mbar_wait_bounded(&full[q % RAW], (q / RAW) & 1u, nullptr, 0);
                return;
            }
            fence_proxy_async_smem();
            fill(k2 + RAW);
        }
    }

    // Each warp takes its share of chunk k + 1's patterns, then adds chunk k's for its trials, so a warp
    // that is late with a chunk holds the others up only when they are one chunk further.
    GsAcc<SW, DPW> acc;
    acc.zero();
    // its share of chunk k's patterns; 0: done, 1: the stream has ended, -1: a wait ran out
    int first = warp;
    auto build = [&](unsigned k) {
        const int s = (int)(k % RAW), b = (int)(k % kGsZ);
        if (!gs_wait(&full[s], (k / RAW) & 1u, a.err)) return -1;
        const int4 m = meta[k % kGsBlobs];
        if (m.w & kGsStop) return 1;
        if (k >= kGsZ && !gs_wait(&added[b], (k / kGsZ - 1) & 1u, a.err)) return -1;
        const int ntasks = (m.y >> 16) & 127;
        const unsigned char *blob = blobs + (k % kGsBlobs) * a.blobcap;
        const int4 *tasks = reinterpret_cast<const int4 *>(blob);
        // the tasks go round the warps from chunk to chunk
        for (int t = first; t < ntasks; t += NW) {
            const int4 h = tasks[t];
            gs_patterns<SW, SIGNED>(reinterpret_cast<const uint4 *>(blob + h.x), h.y & 0xffff, h.y >> 16,
                                    raw + s * a.rawcap, Z + b * a.zcap, h.z, lane, h.w);
        }
        first += first >= kGsTurn ? -kGsTurn : NW - kGsTurn;
        __syncwarp();
        if (lane == 0) mbar_arrive(&built[b]);
        return 0;
    };
    int st = build(0);
    for (unsigned k = 0; st == 0; ++k) {
        st = build(k + 1);
        if (st < 0) break;
        const int b = (int)(k % kGsZ);
        if (!gs_wait(&built[b], (k / kGsZ) & 1u, a.err)) break;
        const int4 m = meta[k % kGsBlobs];
        const int ng = (m.y >> 6) & 31;
        const unsigned char *blob = blobs + (k % kGsBlobs) * a.blobcap;
        gs_add<SW, DPW, NW>(
            acc, Z + b * a.zcap + lane,
            reinterpret_cast<const uint16_t *>(blob + m.z - ng * gs_offsets(NW, DPW) * 2) +
                warp * gs_entry(DPW),
            ng);
        __syncwarp();
        if (lane == 0) mbar_arrive(&added[b]);
        if (m.w & kGsLast) {
            int blk, tile;
            chunks_of(m.x, blk, tile);
            gs_store<SW, DPW, NW>(a, acc, blk, tile, warp, lane);
            acc.zero();
        }
    }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
// Clocks: of a shared-memory wavefront of the patterns and of the adds, of a chunk and of an item; least-
// squares fits to 94 launches (64-4096 channels, 37-4096 trials, 2007-262144 samples), rms errors 3-6%.
struct GsShape {
    int sw, sgn, nw, dpw;
    double build, add, chunk, item;
    const void *fn;
    int db() const { return nw * dpw; }
};
#define GS(S, G, W, D, ...) \
    GsShape{S, G, W, D, __VA_ARGS__, reinterpret_cast<const void *>(&k_group_sum<S, W, D, G>)}
const GsShape kGsShapes[] = {
    GS(1, false, 15, 4, 1.60, 0.95, 1050, 17000), GS(1, false, 19, 2, 1.77, 0.61, 1270, 4400),
    GS(2, false, 15, 4, 0.84, 1.26, 1270, 13500), GS(2, false, 19, 2, 1.36, 0.92, 1280, 5900),
    GS(2, true, 15, 4, 0.84, 1.26, 1270, 13500),  GS(2, true, 19, 2, 1.36, 0.92, 1280, 5900)};
#undef GS

constexpr int kGsTrials = 72;  // trials of a block, at most
constexpr int kGsShare = 8;    // tasks that a chunk aims at (3 and 14 measured 1-8% slower)
constexpr int kGsBlobCap = 2 * 1024;
constexpr int kGsZCap = 58 * 1024 / 4;  // words
constexpr size_t kGsSmem = kGsHead + (size_t)kGsBlobs * kGsBlobCap + kGsZ * (size_t)kGsZCap * 4 +
                           42 * 1024;
static_assert(kGsSmem <= 227 * 1024, "shared memory");
static_assert(kGsZCap < 65536, "16-bit word offsets");

// One group of channels for a block of trials: its distinct patterns (the channels' shifts relative to
// the first's), in an order in which neighbours differ in few rows.
struct GsGroup {
    int c0, n;                       // channels
    int smin, span;                  // of the first channel
    int npats;
    uint64_t pats[kGsTrials];        // a byte per channel: relative shift less lo[i]
    int lo[kGsG];                    // smallest relative shift of a channel
    int nsteps;
    uint8_t pat[kGsTrials];          // a trial's pattern
    bool ok;
};

int popc_bytes(uint64_t x)  // bytes that are not zero
{
    const uint64_t low = 0x7f7f7f7f7f7f7f7full;
    return __builtin_popcountll(((x & low) + low | x) & ~low);
}

// s: the block's first trial's shifts, nd trials of `stride` channels.
void gs_group(const int32_t *s, int nd, long long stride, int c0, int n, GsGroup &q)
{
    q.c0 = c0;
    q.n = n;
    q.ok = true;
    q.npats = 0;
    int rel[kGsTrials][kGsG], lo[kGsG], hi[kGsG];
    int lo0 = INT32_MAX, hi0 = INT32_MIN;
    for (int i = 0; i < kGsG; ++i) {
        lo[i] = INT32_MAX;
        hi[i] = INT32_MIN;
    }
    auto ranges = [&](auto count) {  // (whole groups: a fixed count, which the compiler vectorises)
        const int m = count;
        for (int d = 0; d < nd; ++d) {
            const int32_t *v = s + d * stride + c0;
            lo0 = std::min(lo0, v[0]);
            hi0 = std::max(hi0, v[0]);
            for (int i = 0; i < m; ++i) {
                rel[d][i] = v[i] - v[0];
                lo[i] = std::min(lo[i], rel[d][i]);
                hi[i] = std::max(hi[i], rel[d][i]);
            }
        }
    };
    if (n == kGsG)
        ranges(std::integral_constant<int, kGsG>());
    else
        ranges(n);
    q.smin = lo0;
    q.span = hi0 - lo0;
    for (int i = 0; i < n; ++i) {
        q.lo[i] = lo[i];
        if (hi[i] - lo[i] > 255) q.ok = false;
    }
    if (!q.ok) return;
    uint64_t found[kGsTrials];
    for (int d = 0; d < nd; ++d) {
        uint64_t key = 0;
        for (int i = 1; i < n; ++i) key |= (uint64_t)(uint8_t)(rel[d][i] - lo[i]) << (8 * i);
        int p = d ? q.pat[d - 1] : 0;
        if (!d || found[p] != key)
            for (p = 0; p < q.npats && found[p] != key; ++p) {
            }
        if (p == q.npats) found[q.npats++] = key;
        q.pat[d] = (uint8_t)p;
    }
    // nearest neighbour order
    uint8_t at[kGsTrials];  // old index -> new
    bool used[kGsTrials] = {};
    int cur = 0;
    q.nsteps = (n + 1) / 2;
    for (int k = 0; k < q.npats; ++k) {
        if (k) {
            int best = 99, bi = 0;
            for (int p = 0; p < q.npats; ++p)
                if (!used[p]) {
                    const int diff = popc_bytes(found[p] ^ found[cur]);
                    if (diff < best) {
                        best = diff;
                        bi = p;
                        if (diff == 1) break;
                    }
                }
            q.nsteps += best;
            cur = bi;
        }
        used[cur] = true;
        at[cur] = (uint8_t)k;
        q.pats[k] = found[cur];
    }
    for (int d = 0; d < nd; ++d) q.pat[d] = at[q.pat[d]];
}

int gs_nseg(int sw, int span) { return (kGsT + span + gs_seg(sw) - 1) / gs_seg(sw); }

// Shared-memory wavefronts of a group's patterns, and of the adds that read them.
double gs_build_waves(int sw, const GsGroup &q, int nseg)
{
    return nseg * (9.0 * q.nsteps + (sw == 1 ? 13.0 : 6.0) * (double)q.npats);
}
double gs_add_waves(const GsShape &z) { return z.nw * (z.dpw * (z.sw == 1 ? 8.0 : 16.0) + 1.0); }

// Samples from a staged row's start (the 16-byte boundary below its smallest shift) to where a group's
// first pattern reads row i, less the pattern's own shift of the row.
int gs_row_off(int sw, const GsGroup &q, int i, int smin)
{
    return (smin & (16 / sw - 1)) + q.smin + q.lo[i] - smin;
}

// Bytes of a staged row that hold what is copied and what a group's patterns read of it.
int gs_pitch(int sw, const GsGroup &q, int nseg, const int2 *chan)
{
    int most = 0;
    for (int i = 0; i < q.n; ++i) {
        const int2 ch = chan[q.c0 + i];
        int hi = 0;
        for (int p = 0; p < q.npats; ++p) hi = std::max(hi, (int)(q.pats[p] >> (8 * i) & 255));
        const int read = (gs_row_off(sw, q, i, ch.x) + hi) * sw + (((nseg - 1) * gs_lanes(sw) + 32) * kGsU + 2) * 4;
        const int copied = ((ch.x & (16 / sw - 1)) + kGsT + ch.y) * sw + 16;
        most = std::max(most, std::max(read, copied));
    }
    return kGsPad + (most + 15) / 16 * 16;
}

struct GsChunk {
    size_t g0 = 0, g1 = 0;  // its groups
    int rows = 0, span = 0, nseg = 0, pitch = 0, npats = 0;
    int maxruns = 0, maxsteps = 0;  // with the shortest runs
};

// Whether chunk k with group q more stays within the stage, the pattern buffer and the tables' entry
// (a chunk of one group has to as well: a group that does not fit alone is cut).
bool gs_fits(const GsShape &z, GsChunk &k, const GsGroup &q, const int2 *chan)
{
    const int sw = z.sw;
    GsChunk t = k;
    t.span = std::max(k.span, q.span);
    t.nseg = gs_nseg(sw, t.span);
    t.rows += q.n;
    t.npats += q.npats;
    const int runs = (q.npats + kGsRunMin - 1) / kGsRunMin;
    t.maxruns += runs;
    t.maxsteps += q.nsteps + (runs - 1) * (q.n + 1) / 2;
    t.g1 = k.g1 + 1;
    const int ng = (int)(t.g1 - t.g0);
    // (the pitch of the groups that are in grows with the segments)
    t.pitch = std::max(k.pitch + (t.nseg - k.nseg) * (k.nseg ? gs_lanes(sw) * kGsU * 4 : 0),
                       gs_pitch(sw, q, t.nseg, chan));
    t.pitch = (t.pitch + 15) / 16 * 16;
    if (t.rows > kGsRows || ng > kGsGroups || t.nseg > 31 || t.maxruns * t.nseg > kGsTasks || t.pitch > 255 * 16 ||
        t.rows * t.pitch > gs_rawcap(sw) || t.npats * gs_row_words(sw, t.span) > kGsZCap ||
        16 * (t.maxruns * t.nseg + t.maxsteps) + 2 * gs_offsets(z.nw, z.dpw) * ng > kGsBlobCap)
        return false;
    k = t;
    return true;
}

// The groups of channels [c0, c0 + n): one, or two halves' where those cost less or it does not fit.
double gs_cut(const GsShape &z, const int32_t *s, int nd, long long stride, int c0, int n,
              const int2 *chan, std::vector<GsGroup> &out)
{
    const int sw = z.sw;
    GsGroup q;
    gs_group(s, nd, stride, c0, n, q);
    bool fits = q.ok;
    for (int i = 0; fits && i < n; ++i) {
        const int2 ch = chan[c0 + i];
        fits = gs_row_off(sw, q, i, ch.x) * sw >= -kGsPad;
    }
    const double add = gs_add_waves(z);
    double cost = 0, least = 0;
    if (fits) {
        GsChunk k;
        fits = gs_fits(z, k, q, chan);
        cost = gs_build_waves(sw, q, k.nseg) + add;
        // what a half takes at least: its rows once, one pattern, the adds
        least = gs_nseg(sw, 0) * (9.0 * ((n / 2 + 1) / 2) + (sw == 1 ? 13.0 : 6.0)) + add;
    }
    if (n == 1 || (fits && cost <= 2 * least)) {
        out.push_back(std::move(q));
        return fits ? cost : -1;
    }
    std::vector<GsGroup> a;
    const double l = gs_cut(z, s, nd, stride, c0, n / 2, chan, a);
    const double r = l < 0 || (fits && cost <= l + least)
                         ? -1 : gs_cut(z, s, nd, stride, c0 + n / 2, n - n / 2, chan, a);
    if (r < 0 && !fits) return -1;
    if (r < 0 || (fits && cost <= l + r)) {
        out.push_back(std::move(q));
        return cost;
    }
    for (auto &x : a) out.push_back(std::move(x));
    return l + r;
}

// The shifts' ranges, groups and chunks of the DM block that starts at trial d0.  False where a
// channel's span does not fit.
bool gs_block(const StageGeom &g, const std::vector<int32_t> &S, const GsShape &z, int d0, int2 *chan,
              std::vector<GsGroup> &groups, std::vector<GsChunk> &chunks)
{
    const int nd = std::min(g.ndms - d0, z.db());
    const int32_t *s = &S[(size_t)d0 * g.nchans];
    for (int c = 0; c < g.nchans; ++c) chan[c] = make_int2(s[c], s[c]);
    for (int d = 1; d < nd; ++d) {
        const int32_t *v = s + (size_t)d * g.nchans;
        for (int c = 0; c < g.nchans; ++c)
            chan[c] = make_int2(std::min(chan[c].x, v[c]), std::max(chan[c].y, v[c]));
    }
    for (int c = 0; c < g.nchans; ++c) chan[c].y -= chan[c].x;
    groups.clear();
    chunks.clear();
    for (int c = 0; c < g.nchans; c += kGsG)
        if (gs_cut(z, s, nd, g.nchans, c, std::min(kGsG, g.nchans - c), chan, groups) < 0)
            return false;
    for (size_t i = 0; i < groups.size(); ++i) {
        if (chunks.empty() || !gs_fits(z, chunks.back(), groups[i], chan)) {
            GsChunk k;
            k.g0 = k.g1 = i;
            if (!gs_fits(z, k, groups[i], chan)) return false;
            chunks.push_back(k);
        }
    }
    return true;
}

double gs_block_clocks(const GsShape &z, const std::vector<GsGroup> &groups,
                       const std::vector<GsChunk> &chunks)
{
    double clk = 0;
    for (const GsChunk &k : chunks) {
        for (size_t i = k.g0; i < k.g1; ++i)
            clk += z.build * gs_build_waves(z.sw, groups[i], k.nseg) + z.add * gs_add_waves(z);
        clk += z.chunk;
    }
    return clk;
}

}  // namespace

void gs_release(GsStage &t)
{
    if (t.d_tab) cudaFree(t.d_tab);
    t = GsStage();
}

// Clocks of a launch over `items` tiles, each cut into `split` parts of the channels; the last of the
// waves may be of the costliest blocks.
static double gs_clocks(const GsStage &t, double items, int split, int sms)
{
    return (std::ceil(items * split / sms) - 1.0) * (t.block_clocks / split + kGsShapes[t.shape].item) +
           t.most_clocks / split + kGsShapes[t.shape].item + 11000.0 + (split > 1 ? 5000.0 : 0.0);
}
static int gs_split(const GsStage &t, double items)
{
    int best = 1;
    const int sms = device_sms();
    double clk = gs_clocks(t, items, 1, sms);
    for (int split = 2; split <= 32 && split <= t.min_chunks; ++split) {
        const double c = gs_clocks(t, items, split, sms);
        if (c < 0.95 * clk) {
            clk = c;
            best = split;
        }
    }
    return best;
}

// f(0 .. n-1), each once, on up to eight threads (one for a table so small that a thread costs more).  An f
// that throws (no memory) is one that did nothing.
template <class F>
static void gs_parallel(int n, size_t table, const F &f)
{
    std::atomic<int> next(0);
    auto work = [&]() {
        for (int i = next++; i < n; i = next++) {
            try {
                f(i);
            } catch (...) {
            }
        }
    };
    std::vector<std::thread> pool;
    const int most = table < (1u << 13) ? 1 : std::min({8, (int)std::thread::hardware_concurrency(), n});
    try {
        for (int k = 1; k < most; ++k) pool.emplace_back(work);
    } catch (...) {  // (no more threads: fewer do it)
    }
    work();
    for (auto &p : pool) p.join();
}

// Chooses between the shapes and the shared-memory kernel that est_clocks is of by their estimates: this
// form where it is estimated at 0.9 (16-bit samples 0.85) of the other's time or less.  The uint8 kernels'
// estimate lacks the launches, 16000 clocks; the 16-bit ones' is 8-16 % high instead.  Of 47 measured plans
// it took 23, at 0.47-0.96 of the time; it loses where few channels make wide ones, whose trials hardly
// share patterns.
mdsm_status gs_build(StageGeom &g, const std::vector<int32_t> &S)
try {
    gs_release(g.gs);
    const int sw = (int)dtype_size(g.in_dtype);
    if (g.fixed || g.ngroups != 1 || g.out_u16 || !g.acc_int || sw > 2 ||
        (long long)g.nchans * (sw == 1 ? 255 : 65535) > 0x7fffffffLL)
        return MDSM_OK;
    // the shape by its estimate over (some of) its DM blocks
    auto limit = [&](double other) { return sw == 1 ? 0.9 * (other + 16000.0) : 0.85 * other; };
    double best = limit(g.est_clocks);
    struct Block {  // a DM block's tables in the making
        std::vector<int2> chan;
        std::vector<GsGroup> groups;
        std::vector<GsChunk> chunks;
        double clk = 0;
        bool ok = false;
        void form(const StageGeom &g, const std::vector<int32_t> &S, const GsShape &z, int d0)
        {
            chan.resize((size_t)g.nchans);
            if (!gs_block(g, S, z, d0, chan.data(), groups, chunks)) return;
            clk = gs_block_clocks(z, groups, chunks);
            ok = true;
        }
    };
    struct Sampled {  // a shape, its number of blocks, and every step-th of them
        int shape, nblk, step;
        std::vector<Block> seen;
    };
    std::vector<Sampled> shapes;
    std::vector<std::pair<int, int>> work;
    for (int i = 0; i < (int)(sizeof kGsShapes / sizeof kGsShapes[0]); ++i) {
        const GsShape &z = kGsShapes[i];
        if (z.sw != sw || (z.sgn != 0) != (g.in_dtype == MDSM_I16)) continue;
        const int nblk = (g.ndms + z.db() - 1) / z.db(), step = (nblk + 7) / 8;
        const int n = (nblk + step - 1) / step;
        for (int k = 0; k < n; ++k) work.emplace_back((int)shapes.size(), k);
        shapes.push_back({i, nblk, step, std::vector<Block>((size_t)n)});
    }
    gs_parallel((int)work.size(), S.size(), [&](int w) {
        Sampled &u = shapes[(size_t)work[(size_t)w].first];
        const int k = work[(size_t)w].second;
        const GsShape &z = kGsShapes[u.shape];
        u.seen[(size_t)k].form(g, S, z, k * u.step * z.db());
    });
    GsStage t;
    Sampled *from = nullptr;
    for (Sampled &v : shapes) {
        double clk = 0, most = 0;
        int least = INT32_MAX;
        bool ok = true;
        for (const Block &o : v.seen) {
            ok = ok && o.ok;
            clk += o.clk;
            most = std::max(most, o.clk);
            least = std::min(least, (int)o.chunks.size());
        }
        if (!ok) continue;
        GsStage u;
        u.shape = v.shape;
        u.nblk = v.nblk;
        u.DB = kGsShapes[v.shape].db();
        u.T = kGsT;
        u.block_clocks = clk / (double)v.seen.size();
        u.most_clocks = most;
        u.min_chunks = least;
        const double items = (double)u.nblk * ((g.nsamp + kGsT - 1) / kGsT);
        const double c = gs_clocks(u, items, g.may_split ? gs_split(u, items) : 1, device_sms());
        if (c < best) {
            best = c;
            t = u;
            from = &v;
        }
    }
    if (t.shape < 0) return MDSM_OK;
    const GsShape &z = kGsShapes[t.shape];
    t.chan.resize((size_t)t.nblk * g.nchans);
    // the tables, DM block by DM block, on a few threads (the blocks that were looked at are there)
    struct Table {
        std::vector<uint4> blobs;
        std::vector<int4> chunks;
        double clk = 0;
        bool ok = false;
    };
    std::vector<Table> tables((size_t)t.nblk);
    gs_parallel(t.nblk, S.size(), [&](int b) {
        Block made;
        Block &src = b % from->step == 0 ? from->seen[(size_t)(b / from->step)] : made;
        Table &o = tables[(size_t)b];
        const int d0 = b * t.DB, nd = std::min(g.ndms - d0, t.DB);
        if (!src.ok) src.form(g, S, z, d0);
        if (!src.ok) return;
        int2 *ch = &t.chan[(size_t)b * g.nchans];
        std::copy(src.chan.begin(), src.chan.end(), ch);
        const std::vector<GsGroup> &groups = src.groups;
        const std::vector<GsChunk> &chunks = src.chunks;
        o.clk = src.clk;
        for (const GsChunk &k : chunks) {
            const int ng = (int)(k.g1 - k.g0), rw = gs_row_words(sw, k.span);
            // the groups' patterns in runs, so that about kGsShare warps have a task (each run starts
            // from the rows again)
            const int per = std::max(1, (kGsShare + ng * k.nseg / 2) / (ng * k.nseg));
            std::vector<uint4> runs, st;
            std::vector<uint16_t> offs((size_t)ng * gs_offsets(z.nw, z.dpw), 0);
            int zat = 0, row = 0;
            for (int gi = 0; gi < ng; ++gi) {
                const GsGroup &q = groups[k.g0 + gi];
                auto off = [&](int i, size_t p) {
                    return (unsigned)((row + i) * k.pitch + kGsPad +
                                      (gs_row_off(sw, q, i, ch[q.c0 + i].x) +
                                       (int)(q.pats[p] >> (8 * i) & 255)) * sw);
                };
                auto put = [&](unsigned x, unsigned y, unsigned flag) {
                    st.push_back(make_uint4(x & ~3u, y & ~3u,
                                            x % 4 * 8 | (y % 4 * 8) << 8 | flag << 16, kGsNone));
                };
                const size_t np = (size_t)q.npats;
                const size_t len = std::max<size_t>(kGsRunMin, (np + per - 1) / per);
                for (size_t p = 0; p < np; ++p) {
                    if (p % len == 0) {
                        runs.push_back(make_uint4((unsigned)st.size(), 0, (unsigned)(q.n + 1) / 2, 0));
                        for (int i = 0; i < q.n; i += 2)
                            put(off(i, p), off(std::min(i + 1, q.n - 1), p), i + 1 == q.n);
                    } else {
                        const uint64_t diff = q.pats[p] ^ q.pats[p - 1];
                        for (int i = 0; i < q.n; ++i)
                            if (diff >> (8 * i) & 255) put(off(i, p), off(i, p - 1), 0);
                    }
                    st.back().w = (unsigned)(zat + (int)p * rw);
                    runs.back().y = (unsigned)st.size() - runs.back().x;
                }
                for (int d = 0; d < t.DB; ++d) {
                    int v = zat;
                    if (d < nd) {
                        const int e = S[(size_t)(d0 + d) * g.nchans + q.c0] - q.smin;
                        v += q.pat[d] * rw + (sw == 1 ? (e & 1) * (rw / 2) + e / 2 : e);
                    }
                    offs[(size_t)gi * gs_offsets(z.nw, z.dpw) + d / z.dpw * gs_entry(z.dpw) +
                         d % z.dpw] = (uint16_t)v;
                }
                zat += q.npats * rw;
                row += q.n;
            }
            const size_t at = o.blobs.size();
            const unsigned st0 = (unsigned)runs.size() * k.nseg * 16;  // bytes before the steps
            for (const uint4 &r : runs)
                for (int seg = 0; seg < k.nseg; ++seg)
                    o.blobs.push_back(make_uint4(st0 + r.x * 16, r.y | r.z << 16, (unsigned)seg,
                                                 (unsigned)(sw == 1 ? rw / 2 : rw)));
            o.blobs.insert(o.blobs.end(), st.begin(), st.end());
            const uint4 *ou = reinterpret_cast<const uint4 *>(offs.data());
            o.blobs.insert(o.blobs.end(), ou, ou + offs.size() / 8);
            o.chunks.push_back(make_int4((int)at, (int)(o.blobs.size() - at) * 16, groups[k.g0].c0,
                                         k.rows | ng << 6 | (int)runs.size() * k.nseg << 16 |
                                             k.pitch / 16 << 23));
        }
        o.ok = true;
    });
    t.chunk0.push_back(0);
    t.block_clocks = 0;
    for (const Table &o : tables) {
        const size_t at = t.blobs.size();
        if (!o.ok || at + o.blobs.size() > 0x7fffffffu) return MDSM_OK;
        t.blobs.insert(t.blobs.end(), o.blobs.begin(), o.blobs.end());
        for (int4 k : o.chunks) {
            k.x += (int)at;
            t.chunks.push_back(k);
        }
        t.chunk0.push_back((int)t.chunks.size());
        t.block_clocks += o.clk / t.nblk;
        t.most_clocks = std::max(t.most_clocks, o.clk);
        t.min_chunks = std::min(t.min_chunks, (int)o.chunks.size());
    }
    t.smem = kGsSmem;
    // A launch that folds moments has one part, and may be slower than the packed kernel's where the choice
    // fell for the parts: the same rule again, for one part of both (1734 channels x 3852 samples x 575 trials:
    // 331 us against 238; 192 x 3396 x 25: 46 against 29; whole tiles enough, 801 x 20000 x 300: 281, 329).
    t.whole = gs_clocks(t, (double)t.nblk * ((g.nsamp + kGsT - 1) / kGsT), 1, device_sms()) <
              limit(g.est_whole);
    g.gs = std::move(t);
    return MDSM_OK;
} catch (const std::bad_alloc &) {  // (no memory for these tables on the host either)
    gs_release(g.gs);
    return MDSM_OK;
}

mdsm_status gs_upload(GsStage &t)
{
    if (t.shape < 0) return MDSM_OK;
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t b0 = up(t.blobs.size() * 16), b1 = up(t.chunks.size() * sizeof(int4));
    const size_t b2 = up(t.chunk0.size() * 4), b3 = up(t.chan.size() * sizeof(int2));
    if (cudaMalloc(&t.d_tab, b0 + b1 + b2 + b3) != cudaSuccess) {
        cudaGetLastError();  // (no memory for these tables: the packed kernel runs the stage)
        t = GsStage();
        return MDSM_OK;
    }
    char *d = static_cast<char *>(t.d_tab);
    t.o_chunks = b0;
    t.o_chunk0 = b0 + b1;
    t.o_chan = b0 + b1 + b2;
    MDSM_CUDA_TRY(cudaMemcpy(d, t.blobs.data(), t.blobs.size() * 16, cudaMemcpyHostToDevice));
    MDSM_CUDA_TRY(cudaMemcpy(d + t.o_chunks, t.chunks.data(), t.chunks.size() * sizeof(int4),
                             cudaMemcpyHostToDevice));
    MDSM_CUDA_TRY(cudaMemcpy(d + t.o_chunk0, t.chunk0.data(), t.chunk0.size() * 4,
                             cudaMemcpyHostToDevice));
    MDSM_CUDA_TRY(cudaMemcpy(d + t.o_chan, t.chan.data(), t.chan.size() * sizeof(int2),
                             cudaMemcpyHostToDevice));
    std::vector<uint4>().swap(t.blobs);  // (the device has them)
    std::vector<int4>().swap(t.chunks);
    std::vector<int>().swap(t.chunk0);
    std::vector<int2>().swap(t.chan);
    return MDSM_OK;
}

mdsm_status gs_launch(const StageGeom &g, const void *in, long long in_stride, void *out,
                      long long out_stride, unsigned *d_err, cudaStream_t st, long long nsamp,
                      unsigned long long *mom)
{
    const GsStage &t = g.gs;
    const GsShape &z = kGsShapes[t.shape];
    const char *d = static_cast<const char *>(t.d_tab);
    GsArgs a;
    std::memset(&a, 0, sizeof a);
    a.in = static_cast<const unsigned char *>(in);
    a.in_stride = in_stride;
    a.out = static_cast<unsigned char *>(out);
    a.out_stride = out_stride;
    a.blobs = reinterpret_cast<const uint4 *>(d);
    a.chunks = reinterpret_cast<const int4 *>(d + t.o_chunks);
    a.chunk0 = reinterpret_cast<const int *>(d + t.o_chunk0);
    a.chan = reinterpret_cast<const int2 *>(d + t.o_chan);
    a.nchans = g.nchans;
    a.ndms = g.ndms;
    a.nsamp = (int)nsamp;
    a.nblk = t.nblk;
    const long long ntiles = (nsamp + kGsT - 1) / kGsT;
    a.nsplit = mom || !g.may_split ? 1 : gs_split(t, (double)t.nblk * (double)ntiles);
    const long long nitems = (long long)t.nblk * ntiles * a.nsplit;
    if (nitems > 0x7fffffffLL - 65536) return fail(MDSM_EINVAL, "block too long for one launch");
    a.ntiles = (int)ntiles;
    a.nitems = (int)nitems;
    a.rawcap = gs_rawcap(z.sw);
    a.blobcap = kGsBlobCap;
    a.zcap = kGsZCap;
    a.out_i32 = g.out_i32;
    a.err = d_err;
    a.mom = mom;
    if (a.nsplit > 1)  // the parts add to zeros
        MDSM_CUDA_TRY(cudaMemset2DAsync(out, (size_t)out_stride * 4, 0, (size_t)nsamp * 4,
                                        (size_t)g.ndms, st));
    MDSM_CUDA_TRY(cudaFuncSetAttribute(z.fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kGsSmem));
    void *args[] = {&a};
    const unsigned grid = (unsigned)std::min<long long>(device_sms(), nitems);
    MDSM_CUDA_TRY(cudaLaunchKernel(z.fn, dim3(grid), dim3((unsigned)(z.nw + 1) * 32), args, kGsSmem, st));
    return MDSM_OK;
}

}  // namespace mdsm
