// tmsum.cu -- shift-and-sum of float samples through tensor memory, for brute-force dedispersion and
// both subband stages (the sums of dedisp.cu's generic kernel, channel by channel in the same
// order: the same bits).
//
// A shift-and-sum reads every staged sample once per DM trial.  Shared memory gives 32 words a
// clock per SM, which bounds a kernel that reads one float per add at 32 adds a clock (the generic
// kernel: 29).  Tensor memory gives about 3 times as many (measured: 2.8-3.1 registers per warp and
// clock per SM with 16 columns a load, at any first column), and a load may start at any column,
// which is exactly a shift: lane l of the CTA's 128 tensor-memory lanes holds the samples of time
// segment l, one sample a column, with the halo that the DM block's shifts need, and a trial with
// relative shift e reads the columns from e on.
//
// One CTA: a block of 4 * TPW DM trials x 128 * 12 samples.  A copying warp stages chunks of channels
// (the rows' segments by bulk copies, and the chunk's column offsets) into a ring in shared memory.
// Eight writing warps, two per quarter of the lanes, put a chunk's rows into one half of the columns;
// sixteen adding warps, four per quarter, add it from there for their TPW trials each, while the next
// chunk is written into the other half.  The quarters do not wait for one another, and the chunks of
// consecutive items form one stream, so copies and writes run ahead across items.
//
// What bounds it: the adding warps' loads.  Per trial and channel of a CTA the four quarters load
// 64 registers, 21 clocks at the measured rate, and the kernel takes 27 (16 trials a block, narrow
// spans): without any writing it is only 7% faster.  12 samples a lane (of 16 columns loaded) keep
// the lanes' rows free of bank conflicts (48 bytes apart) and 16 adding warps within the registers;
// 8 or 12 adding warps with more loads a wait measured 10-14% slower, 4 writing warps 2-8%.
// 256 channels x 32344 samples x 500 trials, spans of 3 samples a block: 512 us by the generic
// kernel, 290 here (14.3 Tadd/s).  Wide spans cost columns, and columns chunks: see tm_build.
//
// Column budget: two halves of 256 columns, each 240 for a chunk's channels and 16 of zeros, which
// the padding of a chunk's channel count reads.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>

#include "box.cuh"
#include "internal.h"
#include "ptx.cuh"

namespace mdsm {

namespace {

constexpr int kTmHalf = 256;              // columns of one buffer,
constexpr int kTmBuf = 240;               // of which a chunk's channels take these
constexpr int kTmZero = kTmBuf;           // and the rest are zeros
constexpr int kTmStages = 8;              // chunks in the ring of rows, at most
constexpr int kTmEntries = 8;             // chunks in the ring of headers and offsets (a power of 2)
constexpr int kTmChans = 16;              // channels of a chunk, at most
constexpr int kTmPad = 2;                 // a chunk's channel count is padded to a multiple
constexpr int kTmMain = 16;               // adding warps; then eight that write, one that copies
constexpr int kTmFill = 8;
constexpr int kTmThreads = (kTmMain + kTmFill + 4) * 32;  // (and three idle ones: whole warpgroups)
constexpr int kTmHead = 384;              // barriers, the tensor-memory address
constexpr int kTmMeta = 16 + 4 * kTmChans;  // bytes of a stage's header
constexpr int kTmLast = 1, kTmStop = 2;   // chunk flags
constexpr int kTmL = 12, kTmT = 128 * kTmL;  // samples of a lane, of a tile
constexpr int kTmUnit = 8;                // columns a write moves

// Bytes of a chunk's offsets: a bulk copy moves multiples of 16.
__host__ __device__ constexpr unsigned tm_offbytes(int db, int ncpad)
{
    return (unsigned)(db * ncpad * 2 + 15) / 16 * 16;
}

template <int TPW_>
struct TmCfg {
    static constexpr int TPW = TPW_;  // trials of a warp
    static constexpr int DB = kTmMain / 4 * TPW;
};

}  // namespace

struct TmArgs {
    const unsigned char *in;
    long long in_stride, in_group_stride;    // elements
    float *out;
    long long out_stride, out_group_stride;  // elements
    const uint16_t *offs;   // per chunk [DB][ncpad] column offsets in its buffer
    const int4 *chunks;     // first channel, channels, padded channels, first offset / 8
    const int *chunk0;      // [ngroups * nblk + 1] first chunk of a (group, DM block)
    const int2 *chan;       // [g][blk][c]: smallest shift; column | units << 9 | span << 16
    int nchans, ndms, nsamp, nblk, ntiles, nitems;
    int rowcap;             // bytes of a staged row
    int ncmax;              // channels of the largest chunk
    int nst;                // chunks in the ring
    unsigned *err;
};

namespace {

// A channel's row (src: the lane's samples of it in shared memory) to the columns from `col` on, in
// units of 8 samples.  Two units at a time, so that one's loads overlap the other's stores.
__device__ __forceinline__ void tm_fill_units(const unsigned char *src, uint32_t col, int units)
{
    auto put = [&](uint32_t at, const uint4 &a, const uint4 &b) {
        const uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        tmem_st8(at, v);
    };
    auto get = [&](const unsigned char *p, uint4 &a, uint4 &b) {
        a = *reinterpret_cast<const uint4 *>(p);
        b = *reinterpret_cast<const uint4 *>(p + 16);
    };
    uint4 a0, b0, a1, b1;
    int u = 0;
#pragma unroll 1
    for (; u + 2 <= units; u += 2) {
        get(src, a0, b0);
        get(src + 32, a1, b1);
        put(col, a0, b0);
        put(col + 8, a1, b1);
        src += 64;
        col += 16;
    }
    if (u < units) {
        get(src, a0, b0);
        put(col, a0, b0);
    }
}

template <class C>
struct TmAcc {
    float2 a[C::TPW][kTmL / 2];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int j = 0; j < C::TPW; ++j)
#pragma unroll
            for (int r = 0; r < kTmL / 2; ++r) a[j][r] = make_float2(0.f, 0.f);
    }
};

// One channel's columns added to a trial's sums: channel by channel in order, as the sequential
// sum (a padded channel adds +0 to a sum that is never -0: it starts as +0).
template <class C>
__device__ __forceinline__ void tm_add(TmAcc<C> &acc, int j, const uint32_t *w)
{
#pragma unroll
    for (int r = 0; r < kTmL / 2; ++r)
        acc.a[j][r] = add_f2(acc.a[j][r], make_float2(__uint_as_float(w[2 * r]),
                                                      __uint_as_float(w[2 * r + 1])));
}

// Adds a chunk's channels for the warp's trials.  tb: the buffer's first column (with the
// quarter's lanes); offs: this warp's offsets [TPW][ncpad].  Two channels a wait, the next two's
// offsets loaded before it.  (One channel's loads kept in flight while the one before is added
// measured 4% slower: four warps a quarter cover the waits, and pairs of loads stream better.)
template <class C>
__device__ __forceinline__ void tm_main(TmAcc<C> &acc, uint32_t tb, const uint16_t *offs, int ncpad)
{
    const uint32_t *o = reinterpret_cast<const uint32_t *>(offs);
    uint32_t next = *o++;
#pragma unroll
    for (int j = 0; j < C::TPW; ++j) {
#pragma unroll 1
        for (int c = ncpad; c > 0; c -= 2) {
            const uint32_t cur = next;
            next = *o++;  // (one past the last trial's: spare bytes of the stage, not used)
            uint32_t w[32];
            tmem_ld2x16(w, tb + (cur & 0xffffu), tb + (cur >> 16));
            tm_add<C>(acc, j, w);
            tm_add<C>(acc, j, w + 16);
        }
    }
}

// The item's DM block: fastest, and from tile to tile a different one first, so that a CTA does not meet
// the same block, perhaps the costliest, in each of its items.
__device__ __forceinline__ int tm_block(const TmArgs &a, int item, int rest)
{
    return (int)(((unsigned)item + (unsigned)rest) % (unsigned)a.nblk);
}

// Stores the item's rows of this warp.
template <class C>
__device__ __forceinline__ void tm_store(const TmArgs &a, const TmAcc<C> &acc, int item, int q, int tg,
                                         int lane)
{
    const int rest = item / a.nblk, blk = tm_block(a, item, rest);
    const int tile = rest % a.ntiles, g = rest / a.ntiles;
    const long long t0 = (long long)tile * kTmT + (32 * q + lane) * kTmL;
#pragma unroll
    for (int j = 0; j < C::TPW; ++j) {
        const int d = blk * C::DB + tg * C::TPW + j;
        if (d >= a.ndms) continue;  // (the whole warp)
        float *p = a.out + g * a.out_group_stride + (long long)d * a.out_stride + t0;
        if (t0 + kTmL <= a.nsamp && ((uintptr_t)p & 15) == 0) {
#pragma unroll
            for (int r = 0; r < kTmL / 2; r += 2)
                reinterpret_cast<float4 *>(p)[r / 2] = make_float4(
                    acc.a[j][r].x, acc.a[j][r].y, acc.a[j][r + 1].x, acc.a[j][r + 1].y);
        } else {
#pragma unroll
            for (int r = 0; r < kTmL; ++r)
                if (t0 + r < a.nsamp) p[r] = r & 1 ? acc.a[j][r / 2].y : acc.a[j][r / 2].x;
        }
    }
}

// The registers a thread of the calling warpgroup (four warps) may use from here on.  The kernel is
// launched with kTmRegs a thread; the shares of its seven warpgroups add up to that total exactly
// (an increase waits for registers that others give up, and only the launch's are there).
constexpr int kTmRegs = 72, kTmRegsMain = 96, kTmRegsFill = 40, kTmRegsCopy = 40;
static_assert(kTmMain * kTmRegsMain + kTmFill * kTmRegsFill + 4 * kTmRegsCopy <=
                  (kTmMain + kTmFill + 4) * kTmRegs,
              "register shares");
template <int N>
__device__ __forceinline__ void regs_more()
{
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void regs_fewer()
{
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, unsigned *err)
{
    return !__any_sync(0xffffffffu, !mbar_wait_bounded(bar, parity, err, ERR_WAIT_TIMEOUT));
}

template <class C>
__global__ void __launch_bounds__(kTmThreads, 1)
    k_shift_sum_tm(const __grid_constant__ TmArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    // a chunk's copies have landed / its rows are written to the columns / its offsets are used; a
    // half of a quarter's columns is written / read
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + kTmStages;
    uint64_t *used = empty + kTmStages;
    uint64_t *tfull = used + kTmEntries, *tempty = tfull + 8;  // [2][4]
    uint32_t *slot = reinterpret_cast<uint32_t *>(tempty + 8);
    unsigned char *meta = smem + kTmHead;  // the chunks' headers
    unsigned char *raw = smem + kTmHead + (kTmEntries * kTmMeta + 127) / 128 * 128;
    const unsigned nst = (unsigned)a.nst;
    const int ncpadmax = (a.ncmax + kTmPad - 1) / kTmPad * kTmPad;
    const unsigned rawstage = (unsigned)(a.ncmax * a.rowcap);
    unsigned char *offsm = raw + nst * rawstage + 128;  // (a unit may be read past a row)
    const unsigned offstage = tm_offbytes(C::DB, ncpadmax) + 16;  // (the adds read a word past)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q = warp & 3;

    if (tid == 0) {
        for (unsigned s = 0; s < nst; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kTmFill);
        }
        for (int i = 0; i < kTmEntries; ++i) mbar_init(&used[i], kTmMain);
        for (int i = 0; i < 8; ++i) {
            mbar_init(&tfull[i], kTmFill / 4);
            mbar_init(&tempty[i], kTmMain / 4);
        }
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc_all(slot);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = *slot;
    const uint32_t tq = tmem + ((uint32_t)q << 21);  // the quarter's first lane

    if (warp < kTmMain) {
        // ---- the adds ----
        regs_more<kTmRegsMain>();
        const int tg = warp >> 2;
        TmAcc<C> acc;
        acc.zero();
        for (unsigned k = 0;; ++k) {
            const unsigned buf = k & 1u, e = k & (kTmEntries - 1);
            if (!warp_wait(&tfull[4 * buf + q], (k >> 1) & 1u, a.err)) break;
            tmem_fence_after();
            const int4 h = *reinterpret_cast<const int4 *>(meta + e * kTmMeta);
            if (h.w & kTmStop) break;
            tm_main<C>(acc, tq + buf * kTmHalf,
                       reinterpret_cast<const uint16_t *>(offsm + e * offstage) +
                           tg * C::TPW * h.z, h.z);
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&tempty[4 * buf + q]);
                mbar_arrive(&used[e]);
            }
            if (h.w & kTmLast) {
                tm_store<C>(a, acc, h.x, q, tg, lane);
                acc.zero();
            }
        }
    } else if (warp < kTmMain + kTmFill) {
        // ---- the writes of the quarter's columns ----
        regs_fewer<kTmRegsFill>();
        {
            const uint32_t z[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
            for (int i = 0; i < 4; ++i)
                tmem_st8(tq + (i >> 1) * kTmHalf + kTmZero + (i & 1) * 8, z);
        }
        const int fg = (warp - kTmMain) >> 2;  // the quarter's writing warps take channels in turn
        unsigned s = 0, par = 0;
        for (unsigned k = 0;; ++k) {
            const unsigned buf = k & 1u;
            if (!warp_wait(&full[s], par, a.err)) break;
            if (k >= 2 && !warp_wait(&tempty[4 * buf + q], ((k >> 1) - 1) & 1u, a.err)) break;
            tmem_fence_after();
            const unsigned char *entry = meta + (k & (kTmEntries - 1)) * kTmMeta;
            const int4 h = *reinterpret_cast<const int4 *>(entry);
            const int *mch = reinterpret_cast<const int *>(entry + 16);
            const unsigned char *row =
                raw + s * rawstage + (unsigned)(fg * a.rowcap + (32 * q + lane) * (kTmL * 4));
            for (int i = fg; i < h.y; i += kTmFill / 4, row += kTmFill / 4 * a.rowcap) {
                const int y = mch[i], units = (y >> 9) & 127;
                uint32_t col = tq + buf * kTmHalf + (uint32_t)(y & 511);
                const unsigned char *p = row;
                tm_fill_units(p, col, units);
            }
            tmem_wait_st();
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&tfull[4 * buf + q]);
                if (!(h.w & kTmStop)) mbar_arrive(&empty[s]);
            }
            if (h.w & kTmStop) break;
            if (++s == nst) {
                s = 0;
                par ^= 1u;
            }
        }
    } else {
        // ---- the copies (the last warpgroup's first warp) ----
        regs_fewer<kTmRegsCopy>();
        if (warp == kTmMain + kTmFill) {
            unsigned s = 0, round = 0, n = 0;  // chunk n's rows go to stage s, round `round` of the ring
            bool late = false;
            // waits for stage s and chunk n's entry to be free again
            auto claim = [&]() {
                if (round > 0 && !warp_wait(&empty[s], (round - 1) & 1u, a.err)) return false;
                if (n >= kTmEntries &&
                    !warp_wait(&used[n & (kTmEntries - 1)], (n / kTmEntries - 1) & 1u, a.err))
                    return false;
                fence_proxy_async_smem();
                return true;
            };
            auto next_stage = [&]() {
                ++n;
                if (++s == nst) {
                    s = 0;
                    ++round;
                }
            };
            for (int it = blockIdx.x; it < a.nitems && !late; it += gridDim.x) {
                const int rest = it / a.nblk, blk = tm_block(a, it, rest);
                const int tile = rest % a.ntiles, g = rest / a.ntiles;
                const long long t0 = (long long)tile * kTmT;
                const int cnt = (int)min((long long)kTmT, (long long)a.nsamp - t0);
                const int gb = g * a.nblk + blk;
                const int2 *chan = a.chan + (size_t)gb * a.nchans;
                const unsigned char *in_g = a.in + (size_t)(g * a.in_group_stride) * 4;
                const int k0 = __ldg(a.chunk0 + gb), k1 = __ldg(a.chunk0 + gb + 1);
                int4 ck = __ldg(a.chunks + k0);
                int2 ch = lane < ck.y ? __ldg(chan + ck.x + lane) : make_int2(0, 0);
                for (int k = k0; k < k1; ++k) {
                    // the next chunk's entries are loaded before this one waits for its stage
                    const int4 nk = k + 1 < k1 ? __ldg(a.chunks + k + 1) : make_int4(0, 0, 0, 0);
                    const int2 nch = lane < nk.y ? __ldg(chan + nk.x + lane) : make_int2(0, 0);
                    if (!claim()) {
                        late = true;
                        break;
                    }
                    unsigned char *entry = meta + (n & (kTmEntries - 1)) * kTmMeta;
                    unsigned bytes = 0;
                    const unsigned char *src = nullptr;
                    if (lane < ck.y) {
                        const long long start = t0 + ch.x;
                        const long long end = start + cnt + ((unsigned)ch.y >> 16);
                        const long long sb = (start * 4) & ~15LL;
                        const long long eb = (end * 4 + 15) & ~15LL;
                        bytes = (unsigned)(eb - sb);
                        src = in_g + (size_t)(ck.x + lane) * (size_t)a.in_stride * 4 + sb;
                        reinterpret_cast<int *>(entry + 16)[lane] = ch.y;
                    }
                    if (lane == 0)
                        *reinterpret_cast<int4 *>(entry) =
                            make_int4(it, ck.y, ck.z, k + 1 == k1 ? kTmLast : 0);
                    const unsigned offbytes = tm_offbytes(C::DB, ck.z);
                    unsigned total = bytes;
    #pragma unroll
                    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
                    __syncwarp();
                    if (lane == 0) mbar_arrive_expect_tx(&full[s], total + offbytes);
                    __syncwarp();
                    if (lane < ck.y)
                        bulk_g2s(raw + s * rawstage + (unsigned)(lane * a.rowcap), src, bytes, &full[s]);
                    if (lane == 0)
                        bulk_g2s(offsm + (n & (kTmEntries - 1)) * offstage, a.offs + (size_t)ck.w * 8,
                                 offbytes, &full[s]);
                    next_stage();
                    ck = nk;
                    ch = nch;
                }
            }
            if (!late && claim()) {  // the end of the stream
                if (lane == 0) {
                    *reinterpret_cast<int4 *>(meta + (n & (kTmEntries - 1)) * kTmMeta) =
                        make_int4(-1, 0, 0, kTmStop);
                    mbar_arrive(&full[s]);
                }
            } else {
                // let the copies already issued land before the CTA exits (bounded as well)
                for (unsigned m = 0; m < nst; ++m)
                    if (m < s || round > 0)
                        mbar_wait_bounded(&full[m], (m < s ? round : round - 1u) & 1u, nullptr, 0);
            }
        }
    }
    __syncwarp();
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    if (warp == 0) tmem_free_all(tmem);
}

}  // namespace

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
namespace {

struct TmShape {
    int tpw;
    const void *fn;
};

#define TM(P) TmShape{P, reinterpret_cast<const void *>(&k_shift_sum_tm<TmCfg<P>>)}
const TmShape kTmShapes[] = {TM(4), TM(3), TM(2)};
#undef TM

// Each launch asks for all of a CTA's shared memory.  With the 1 KB that the system keeps per CTA that is all
// the SM has, so a CTA gets an SM that no other CTA (of any kernel) is on or comes to: the tensor memory is
// free, and its allocation, the one wait here that has no bound, does not wait.
constexpr size_t kTmSmem = 227 * 1024;

// Bytes that a ring of nst chunks needs of it.
size_t tm_smem(int nst, int ncmax, int rowcap, int db)
{
    const int ncpad = (ncmax + kTmPad - 1) / kTmPad * kTmPad;
    return kTmHead + (kTmEntries * kTmMeta + 127) / 128 * 128 + (size_t)nst * ncmax * rowcap + 128 +
           (size_t)kTmEntries * (tm_offbytes(db, ncpad) + 16);
}

}  // namespace

void tm_release(TmStage &t)
{
    if (t.d_tab) cudaFree(t.d_tab);
    t = TmStage();
}

// The smallest and largest shift of every channel over kTmGran trials (which divides each shape's
// blocks), [g][trials / kTmGran][c]: the shapes' tables start from these.
constexpr int kTmGran = 4;
static std::vector<int2> tm_ranges(const StageGeom &g, const std::vector<int32_t> &S)
{
    const int n = (g.ndms + kTmGran - 1) / kTmGran;
    std::vector<int2> r((size_t)g.ngroups * n * g.nchans);
    for (int gi = 0; gi < g.ngroups; ++gi)
        for (int d = 0; d < g.ndms; ++d) {
            const int32_t *s = &S[((size_t)gi * g.ndms + d) * g.nchans];
            int2 *o = &r[((size_t)gi * n + d / kTmGran) * g.nchans];
            if (d % kTmGran == 0)
                for (int c = 0; c < g.nchans; ++c) o[c] = make_int2(s[c], s[c]);
            else
                for (int c = 0; c < g.nchans; ++c)
                    o[c] = make_int2(std::min(o[c].x, s[c]), std::max(o[c].y, s[c]));
        }
    return r;
}

// Tables of shape `sh` for a stage.  False where a channel's columns do not fit a half.
static bool tm_tables(const StageGeom &g, const std::vector<int2> &ranges, int sh, TmStage &t)
{
    const TmShape &z = kTmShapes[sh];
    constexpr int per16 = 4, unit = kTmUnit;
    const int DB = kTmMain / 4 * z.tpw;
    const int nblk = (g.ndms + DB - 1) / DB, ngb = g.ngroups * nblk;
    t.shape = sh;
    t.nblk = nblk;
    t.T = kTmT;
    t.DB = DB;
    t.chan.resize((size_t)ngb * g.nchans);
    t.chunk0.assign((size_t)ngb + 1, 0);
    // the smallest shift and the span of every (DM block, channel)
    int maxspan = 0;
    const int nr = (g.ndms + kTmGran - 1) / kTmGran;
    for (int gi = 0; gi < g.ngroups; ++gi)
        for (int b = 0; b < nblk; ++b) {
            const int r0 = b * DB / kTmGran, r1 = std::min(nr, r0 + DB / kTmGran);
            const int2 *r = &ranges[((size_t)gi * nr + r0) * g.nchans];
            int2 *chan = &t.chan[((size_t)gi * nblk + b) * g.nchans];
            for (int c = 0; c < g.nchans; ++c) {
                int2 v = r[c];
                for (int k = 1; k < r1 - r0; ++k) {
                    const int2 w = r[(size_t)k * g.nchans + c];
                    v = make_int2(std::min(v.x, w.x), std::max(v.y, w.y));
                }
                chan[c] = make_int2(v.x, v.y - v.x);
                maxspan = std::max(maxspan, v.y - v.x);
            }
        }
    if (kTmL + (per16 - 1) + maxspan + unit - 1 > kTmBuf) return false;
    // a staged row: the tile, the span, what precedes smin in its 16 bytes, and a last unit's rest
    t.rowcap = ((kTmT + maxspan + per16 + unit) * 4 + 15) / 16 * 16 + 16;
    // a chunk is a run of channels whose columns fit a buffer and whose rows fit the ring
    int nclim = kTmChans;
    while (nclim > 0 && tm_smem(3, nclim, t.rowcap, DB) > kTmSmem) --nclim;
    if (nclim < 1) return false;
    size_t noff = 0;
    int ncmax = 1;
    std::vector<int> spans((size_t)g.nchans);
    for (int gb = 0; gb < ngb; ++gb) {
        t.chunk0[gb] = (int)t.chunks.size();
        int2 *chan = &t.chan[(size_t)gb * g.nchans];
        int c0 = 0, col = 0;
        for (int c = 0; c < g.nchans; ++c) spans[(size_t)c] = chan[c].y;
        auto close = [&](int c1) {
            const int nc = c1 - c0, ncpad = (nc + kTmPad - 1) / kTmPad * kTmPad;
            t.chunks.push_back(make_int4(c0, nc, ncpad, (int)(noff / 8)));
            noff += ((size_t)DB * ncpad + 7) / 8 * 8;
            ncmax = std::max(ncmax, nc);
        };
        for (int c = 0; c < g.nchans; ++c) {
            const int span = spans[(size_t)c], rem = chan[c].x & (per16 - 1);
            const int units = (kTmL + rem + span + unit - 1) / unit, need = units * unit;
            if (c > c0 && (col + need > kTmBuf || c - c0 == nclim)) {
                // (an even number of channels: the padding would be read like one)
                if (((c - c0) & 1) && c - c0 > 1) --c;
                close(c);
                c0 = c--;
                col = 0;
                continue;
            }
            chan[c].y = col | units << 9 | span << 16;
            col += need;
        }
        close(g.nchans);
    }
    t.chunk0[(size_t)ngb] = (int)t.chunks.size();
    if (noff / 8 > 0x7fffffffull) return false;
    t.ncmax = ncmax;
    // a ring of at least three chunks, more where they fit: short chunks need the lead
    t.nst = 3;
    while (t.nst < kTmStages && tm_smem(t.nst + 1, ncmax, t.rowcap, DB) <= kTmSmem) ++t.nst;
    t.smem = kTmSmem;
    t.noff = noff;
    return true;
}

// Column offsets, chunk by chunk [DB][ncpad]; padded channels and trials read zeros.
static void tm_offsets(const StageGeom &g, const std::vector<int32_t> &S, TmStage &t)
{
    constexpr int per16 = 4;
    t.offs.assign(t.noff, (uint16_t)0);
    for (int gi = 0; gi < g.ngroups; ++gi)
        for (int b = 0; b < t.nblk; ++b) {
            const size_t gb = (size_t)gi * t.nblk + b;
            const int d0 = b * t.DB, d1 = std::min(g.ndms, d0 + t.DB);
            const int2 *chan = &t.chan[gb * g.nchans];
            for (int k = t.chunk0[gb]; k < t.chunk0[gb + 1]; ++k) {
                const int4 ck = t.chunks[(size_t)k];
                uint16_t *o = &t.offs[(size_t)ck.w * 8];
                for (int d = d0; d < d0 + t.DB; ++d, o += ck.z) {
                    const int32_t *s =
                        d < d1 ? &S[((size_t)gi * g.ndms + d) * g.nchans + ck.x] : nullptr;
                    for (int i = 0; i < ck.z; ++i) {
                        if (i >= ck.y || !s) {
                            o[i] = (uint16_t)kTmZero;
                            continue;
                        }
                        const int2 ch = chan[ck.x + i];
                        const int e = (ch.x & (per16 - 1)) + s[i] - ch.x;
                        o[i] = (uint16_t)((ch.y & 511) + e);
                    }
                }
            }
        }
}

// The launch's estimated clocks in this form: 17.4 a trial and channel of a block, 1550 a chunk (its
// channels' last pairs, the waits) and an item, and the launch with its first chunks 15000; a least-squares
// fit to 240 launches (64-4096 channels, 32-3929 trials, 2295-250094 samples, spans of 0-130) with an rms
// error of 8%.
static double tm_clocks(const StageGeom &g, const TmStage &t)
{
    const double items = (double)g.ngroups * t.nblk;
    const double waves = std::ceil(items * ((g.nsamp + kTmT - 1) / kTmT) / device_sms());
    int most = 0;  // (the last wave may be of the blocks with the most chunks)
    for (size_t b = 0; b + 1 < t.chunk0.size(); ++b) most = std::max(most, t.chunk0[b + 1] - t.chunk0[b]);
    return waves * (17.4 * g.nchans * t.DB + 1550.0) +
           1550.0 * ((waves - 1.0) * (double)t.chunks.size() / items + most) + 15000.0;
}

// Whether a shape's kernel came out at the registers whose shares it deals out (its increase would wait for
// ever on fewer).
static bool tm_built(const TmShape &z)
{
    cudaFuncAttributes at;
    if (cudaFuncGetAttributes(&at, z.fn) != cudaSuccess) {
        cudaGetLastError();  // (the generic kernel runs the stage)
        return false;
    }
    return at.numRegs == kTmRegs;
}

// Chooses among the shapes and the generic kernel by their estimates.  This form is taken where it is
// estimated at 0.85 of the generic kernel's time or less, which leaves room for the error of both: of
// 97 measured plans it took 56, at 0.44-0.97 of the generic kernel's time.  It loses where spans are
// wide (1 MHz channels at 1.2 GHz, steps of 1 pc cm^-3: 12 samples a block and more; a chunk is then
// two or three channels) and where there are too few tiles of 1536 samples to fill the SMs.
mdsm_status tm_build(StageGeom &g, const std::vector<int32_t> &S)
try {
    tm_release(g.tm);
    // (int32 output is converted by the generic kernel's store; this one stores floats)
    if (g.in_dtype != MDSM_F32 || g.out_i32 || g.fixed) return MDSM_OK;
    const std::vector<int2> ranges = tm_ranges(g, S);
    double best = 0.85 * g.est_clocks;
    TmStage pick;
    for (int i = 0; i < (int)(sizeof kTmShapes / sizeof kTmShapes[0]); ++i) {
        TmStage t;
        if (!tm_built(kTmShapes[i]) || !tm_tables(g, ranges, i, t)) continue;
        const double clk = tm_clocks(g, t);
        if (clk < best) {
            best = clk;
            pick = std::move(t);
        }
    }
    if (pick.shape < 0) return MDSM_OK;
    tm_offsets(g, S, pick);
    g.tm = std::move(pick);
    return MDSM_OK;
} catch (const std::bad_alloc &) {  // (no memory for these tables on the host either)
    tm_release(g.tm);
    return MDSM_OK;
}

mdsm_status tm_upload(TmStage &t)
{
    if (t.shape < 0) return MDSM_OK;
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t b0 = up(t.offs.size() * 2), b1 = up(t.chunks.size() * sizeof(int4));
    const size_t b2 = up(t.chunk0.size() * 4), b3 = up(t.chan.size() * sizeof(int2));
    if (cudaMalloc(&t.d_tab, b0 + b1 + b2 + b3) != cudaSuccess) {
        cudaGetLastError();  // (no memory for these tables: the generic kernel runs the stage)
        t = TmStage();
        return MDSM_OK;
    }
    char *d = static_cast<char *>(t.d_tab);
    MDSM_CUDA_TRY(cudaMemcpy(d, t.offs.data(), t.offs.size() * 2, cudaMemcpyHostToDevice));
    MDSM_CUDA_TRY(cudaMemcpy(d + b0, t.chunks.data(), t.chunks.size() * sizeof(int4),
                             cudaMemcpyHostToDevice));
    MDSM_CUDA_TRY(cudaMemcpy(d + b0 + b1, t.chunk0.data(), t.chunk0.size() * 4,
                             cudaMemcpyHostToDevice));
    MDSM_CUDA_TRY(cudaMemcpy(d + b0 + b1 + b2, t.chan.data(), t.chan.size() * sizeof(int2),
                             cudaMemcpyHostToDevice));
    t.o_chunks = b0;
    std::vector<uint16_t>().swap(t.offs);  // (the device has them)
    std::vector<int2>().swap(t.chan);
    std::vector<int4>().swap(t.chunks);
    std::vector<int>().swap(t.chunk0);
    t.o_chunk0 = b0 + b1;
    t.o_chan = b0 + b1 + b2;
    return MDSM_OK;
}

mdsm_status tm_launch(const StageGeom &g, const void *in, long long in_stride,
                      long long in_group_stride, void *out, long long out_stride,
                      long long out_group_stride, unsigned *d_err, cudaStream_t st, long long nsamp)
{
    const TmStage &t = g.tm;
    const TmShape &z = kTmShapes[t.shape];
    MDSM_CUDA_TRY(cudaFuncSetAttribute(z.fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)t.smem));
    const char *d = static_cast<const char *>(t.d_tab);
    TmArgs a;
    std::memset(&a, 0, sizeof a);
    a.in = static_cast<const unsigned char *>(in);
    a.in_stride = in_stride;
    a.in_group_stride = in_group_stride;
    a.out = static_cast<float *>(out);
    a.out_stride = out_stride;
    a.out_group_stride = out_group_stride;
    a.offs = reinterpret_cast<const uint16_t *>(d);
    a.chunks = reinterpret_cast<const int4 *>(d + t.o_chunks);
    a.chunk0 = reinterpret_cast<const int *>(d + t.o_chunk0);
    a.chan = reinterpret_cast<const int2 *>(d + t.o_chan);
    a.nchans = g.nchans;
    a.ndms = g.ndms;
    a.nsamp = (int)nsamp;
    a.nblk = t.nblk;
    const long long ntiles = (nsamp + kTmT - 1) / kTmT;
    const long long nitems = (long long)t.nblk * ntiles * g.ngroups;
    if (nitems > 0x7fffffffLL) return fail(MDSM_EINVAL, "block too long for one launch");
    a.ntiles = (int)ntiles;
    a.nitems = (int)nitems;
    a.rowcap = t.rowcap;
    a.ncmax = t.ncmax;
    a.nst = t.nst;
    a.err = d_err;
    void *args[] = {&a};
    const unsigned grid = (unsigned)std::min<long long>(device_sms(), nitems);
    MDSM_CUDA_TRY(cudaLaunchKernel(z.fn, dim3(grid), dim3(kTmThreads), args, t.smem, st));
    return MDSM_OK;
}

}  // namespace mdsm
