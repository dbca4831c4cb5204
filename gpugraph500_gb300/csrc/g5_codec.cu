// g5_codec.cu -- the s4-bp128 frontier-queue codec on the device.
//
// Wire format (identical, word for word, to the reference's vendored
// SIMDCompressionAndIntersection library as configured by the reference,
// cpu_2d/compression/cpusimd/include/codecfactory.h:103-108):
//
//   CompositeCodec (compositecodec.h:31-71): the first floor(n/128)*128 values
//   go to SIMDBinaryPacking, the rest to VariableByte<true>.
//   SIMDBinaryPacking (simdbinarypacking.h:174-289): word 0 = n1, three
//   cookie words 123456, then groups of 16 miniblocks of 128 values: four
//   header words with the 16 bit widths (big-endian bytes), then each
//   miniblock's 4*b payload words.  A partial last group still writes the
//   four header words.
//   Miniblock (SIMDIntegratedBlockPacker, deltatemplates.h:67-120): 32
//   vectors of 4 lanes; d4 subtracts the previous vector lane-wise, dm
//   subtracts lane 3 of the previous vector; the previous vector of the
//   first miniblock is zero; b = bit length of the OR of all deltas; each lane
//   packs its 32 deltas LSB-first, word w of lane l at 4w+l; b = 32 stores the
//   raw values.
//   VariableByte<true> (variablebyte.h:100-161): delta from 0, 7-bit groups
//   little-endian, high bit on the last byte, zero-padded to a word.
//
// GPU design, one stream per call: every miniblock is independent for
// encoding (its deltas only need the input), so one warp packs one miniblock,
// and a chunk's place in the stream is the sum of the word counts that the
// chunks before it publish.
// Decoding needs each group's position, which the stream only gives as a
// chain (each header says how long its group is), and the sums of all values
// before it: one launch, a block per chunk of the stream, which finds its own
// place in the chain and adds up what the chunks before it publish.  The
// many-streams calls run the chunks of all k queues in one launch each way.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "g5_codec_dev.cuh"
#include "g5_common.cuh"

namespace g5 {

namespace {

constexpr uint32_t kCookie = 123456u;
constexpr int kTailMaxBytes = 4096;  // largest VariableByte tail decoded

__device__ __forceinline__ uint32_t bits_of(uint32_t v) { return v ? 32u - __clz(v) : 0u; }

// Running lane sums that a raw miniblock restarts.
struct ResetAdd {
    typedef VecFlag T;
    __device__ static T id()
    {
        T t;
        t.v = make_uint4(0, 0, 0, 0);
        t.f = 0;
        return t;
    }
    __device__ static T op(T a, T b)
    {
        if (b.f) return b;
        T r;
        r.v = make_uint4(a.v.x + b.v.x, a.v.y + b.v.y, a.v.z + b.v.z, a.v.w + b.v.w);
        r.f = a.f;
        return r;
    }
    __device__ static T shfl_up(T v, int o)
    {
        T r;
        r.v.x = __shfl_up_sync(0xFFFFFFFFu, v.v.x, o);
        r.v.y = __shfl_up_sync(0xFFFFFFFFu, v.v.y, o);
        r.v.z = __shfl_up_sync(0xFFFFFFFFu, v.v.z, o);
        r.v.w = __shfl_up_sync(0xFFFFFFFFu, v.v.w, o);
        r.f = __shfl_up_sync(0xFFFFFFFFu, v.f, o);
        return r;
    }
};

// ---- encoder ---------------------------------------------------------------------------

__device__ __forceinline__ uint4 deltas(uint4 cur, uint4 prev, int mode)
{
    if (mode == G5_CODEC_DM)
        return make_uint4(cur.x - prev.w, cur.y - prev.w, cur.z - prev.w, cur.w - prev.w);
    return make_uint4(cur.x - prev.x, cur.y - prev.y, cur.z - prev.z, cur.w - prev.w);
}

// ---- meetings of a launch's blocks -------------------------------------------------------
//
// Blocks claim chunks in launch order from a counter, so a chunk only ever
// waits on chunks claimed before it, whose blocks are already running.  A
// chunk's record holds the call's epoch, so what earlier calls left reads as
// "not published" and nothing is cleared between calls.  The last block to finish
// resets the counter and advances the epoch.  Every wait is bounded: past
// kSpinLimit polls the kernel records G5_DEVERR_WAIT and goes on with what it
// has, so no launch can spin forever.

constexpr uint32_t kSpinLimit = 1u << 21;
enum : uint32_t { ST_NONE = 0, ST_AGG = 1, ST_INC = 2 };

// scalar slots of the two (the scalar block holds kScalars)
enum { CS_E_CTR = 20, CS_E_DONE = 21, CS_E_EPOCH = 22, CS_E_ERR = 23, CS_E_WORDS = 24 };
enum { CS_U_CTR = 25, CS_U_DONE = 26, CS_U_EPOCH = 27, CS_U_ERR = 28, CS_U_N = 29 };

__device__ __forceinline__ uint64_t vload64(const uint64_t *p) { return *reinterpret_cast<const volatile uint64_t *>(p); }
// A 16-byte part of a record and its status, in one access each way: a reader
// needs no fence and no second round trip.
__device__ __forceinline__ void put_part(unsigned long long *p, unsigned long long value, unsigned long long status)
{
    const unsigned __int128 x = (unsigned __int128)status << 64 | value;
    asm volatile("st.relaxed.gpu.global.b128 [%0], %1;\n" ::"l"(__cvta_generic_to_global(p)), "q"(x) : "memory");
}

__device__ __forceinline__ void get_part(const unsigned long long *p, unsigned long long &value,
                                         unsigned long long &status)
{
    unsigned __int128 x;
    asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];\n" : "=q"(x) : "l"(__cvta_generic_to_global(p)) : "memory");
    value = (unsigned long long)x;
    status = (unsigned long long)(x >> 64);
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(__cvta_generic_to_global(gmem)) : "memory");
}

// Claims the next tile for the whole block (thread 0 draws, all read).
__device__ __forceinline__ uint64_t claim_tile(uint64_t *ctr, uint64_t *s_t)
{
    __syncthreads();  // the previous tile's shared state is no longer read
    if (threadIdx.x == 0) *s_t = atomicAdd((unsigned long long *)ctr, 1ull);
    __syncthreads();
    return *s_t;
}

// True in the block that finishes last (thread 0 only); it may then reset the
// call's counters: every other block has passed its last read of them.
__device__ __forceinline__ bool last_block(uint64_t *done)
{
    __syncthreads();
    if (threadIdx.x != 0) return false;
    __threadfence();
    return atomicAdd((unsigned long long *)done, 1ull) == gridDim.x - 1;
}

// Stream header words and the VariableByte tail of n - n1 (< 128) values,
// written by one warp; blkend = word after the block part.  Returns the
// stream's words.  (compositecodec.h:31-51, variablebyte.h:100-161: each
// value's delta from the one before, 0 before the first, in 7-bit groups from
// the low end, the high bit on the last byte, zero-padded to a word.)  One lane
// per value: its byte count, their exclusive prefix over the warp (its place),
// then its bytes.
__device__ uint64_t enc_tail_warp(const uint32_t *in, uint64_t n, uint64_t n1, uint64_t blkend, uint32_t *out,
                                  uint32_t *s_bytes)
{
    const int lane = g5_lane();
    const uint32_t nt = (uint32_t)(n - n1);
    for (uint32_t i = lane; i < (128 * 5 + 3) / 4 + 1; i += 32) s_bytes[i] = 0;
    __syncwarp();
    uint8_t *bb = reinterpret_cast<uint8_t *>(s_bytes);
    uint32_t p = 0, last = 0;  // bytes so far and the value before this round (warp-uniform)
    for (uint32_t i0 = 0; i0 < nt; i0 += 32) {
        const uint32_t i = i0 + lane;
        const bool have = i < nt;
        const uint32_t x = have ? in[n1 + i] : 0u;
        uint32_t px = __shfl_up_sync(0xFFFFFFFFu, x, 1);
        if (lane == 0) px = last;
        const uint32_t d = x - px;
        const uint32_t len = have ? 1u + (d >= (1u << 7)) + (d >= (1u << 14)) + (d >= (1u << 21)) + (d >= (1u << 28)) : 0u;
        uint32_t inc = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += y;
        }
        const uint32_t at = p + inc - len;
        for (uint32_t k = 0; k < len; ++k)
            bb[at + k] = (uint8_t)(((d >> (7 * k)) & 127u) | (k + 1 == len ? 128u : 0u));
        p += __shfl_sync(0xFFFFFFFFu, inc, 31);
        last = __shfl_sync(0xFFFFFFFFu, x, 31);
    }
    __syncwarp();
    const uint32_t tw = (p + 3) / 4;
    if (lane == 0) {
        out[0] = (uint32_t)n1;
        out[1] = kCookie;
        out[2] = kCookie;
        out[3] = kCookie;
    }
    for (uint32_t i = lane; i < tw; i += 32) out[blkend + i] = s_bytes[i];
    return blkend + tw;
}

// ---- encoder ----------------------------------------------------------------------------
//
// One launch.  A miniblock's bit width depends only on its own 128 values and
// the vector before them, so the stream's layout is fixed once every width is
// known.  A block takes a chunk of up to kEG groups (16 miniblocks each),
// claimed in launch order:
//   load    its values into shared memory
//   widths  a warp per miniblock turns its values into deltas, in place, and
//           ORs them
//   meet    the chunk's word count is published (one 16-byte store that carries
//           its own status) and those of up to 512 chunks before it are read
//           at once: the chunk's place in the stream
//   pack    a warp per miniblock gathers each word of the payload from the
//           values that reach into it and stores it, coalesced
// The block with the last group writes the stream header and the VariableByte
// tail.  n may come from device memory: the launch can sit in a CUDA graph with
// a fixed grid.
//
// What bounds it: a chain of round trips (start 1.1 us, load 0.4-0.8, widths and
// their scan 0.8-2.5, meeting 0.7-1.6, the last block's exit 1.3), and on large
// queues issue: widths 1.7 us and packing 3 us of the 13 that 5 M values take
// (23.8 MB of traffic).  The values are read once; the two launches this replaced
// (widths, then packing from a second read with shared-memory atomics) took 18
// us for the same queue, and 5.7 against 3.9 for 3000 values.
constexpr int kEB = 512;  // threads per block
constexpr uint64_t kLoneRaw = 4096;  // values one block copies
constexpr int kEW = kEB / 32;
constexpr int kEG = 8;    // groups per chunk at most (64 KB of values: three blocks per SM)
constexpr int kEM = 16 * kEG;
constexpr uint32_t kSlot = 16;  // 64-bit words from one chunk's record to the next (a line each: all blocks read
                                // all of them at once, and neighbours in one line queue up there)


// Exclusive scan over the block (kEB threads) of a 32-bit value; total -> tot.
__device__ __forceinline__ uint32_t block_excl_u32(uint32_t x, uint32_t *s_w, uint32_t &tot)
{
    const int lane = g5_lane(), wid = threadIdx.x >> 5;
    uint32_t inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) s_w[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const uint32_t v = lane < kEB / 32 ? s_w[lane] : 0u;
        uint32_t vi = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, vi, o);
            if (lane >= o) vi += y;
        }
        if (lane < kEB / 32) s_w[lane] = vi - v;
        if (lane == kEB / 32 - 1) s_w[kEB / 32] = vi;
    }
    __syncthreads();
    const uint32_t r = s_w[wid] + inc - x;
    tot = s_w[kEB / 32];
    __syncthreads();
    return r;
}

struct EncShared {
    uint4 prev[kEM];               // the vector before each miniblock
    uint4 vec[kEM * 32];           // the chunk's values, then their deltas
    uint32_t off[kEM];             // words from the chunk's first header to each miniblock's payload
    __align__(16) uint8_t b[kEM];  // widths
    uint32_t w[kEB / 32 + 1];
    uint64_t t;
    unsigned long long before;     // words before the chunk
    int near_inc;
    uint32_t magic[32];            // 2^16 / b + 1: quotients by b of up to 1023
    uint32_t bytes[(128 * 5 + 3) / 4 + 1];
};

struct EncLen {
    uint64_t n, n1, nmb, ng, nchunks;
    uint32_t gpc;  // groups per chunk
    bool raw, too_long;
};

__device__ __forceinline__ EncLen enc_len(uint64_t n_in, uint64_t max_n, uint64_t raw_thr, uint32_t blocks)
{
    EncLen e;
    e.too_long = n_in > max_n;  // a device-side length past the workspace: nothing is written
    e.n = e.too_long ? 0 : n_in;
    e.nmb = e.n / 128;
    e.n1 = e.nmb * 128;
    e.ng = (e.nmb + 15) / 16;
    // (two groups are one block's, which then waits for nobody)
    e.gpc = e.ng <= 2 ? 2u : (uint32_t)min((uint64_t)kEG, max((uint64_t)1, (e.ng + blocks - 1) / blocks));
    e.nchunks = (e.ng + e.gpc - 1) / e.gpc;
    e.raw = raw_thr && e.n <= raw_thr;
    return e;
}

// Words of the chunks before chunk c, by the whole block, into sh.before.
__device__ void enc_before(EncShared &sh, uint64_t c, uint64_t epoch, const unsigned long long *slots, uint32_t stride,
                           uint64_t *err)
{
    if (threadIdx.x == 0) sh.before = 0;
    for (int64_t hi = (int64_t)c - 1; hi >= 0; hi -= kEB) {
        if (threadIdx.x == 0) sh.near_inc = kEB;
        __syncthreads();
        const int64_t j = hi - threadIdx.x;
        unsigned long long x = 0, t = 0;
        if (j >= 0) {
            uint32_t spins = 0;
            for (;;) {
                get_part(slots + stride * j, x, t);
                if ((t >> 2) == epoch && (t & 3)) break;
                if (++spins > kSpinLimit) {
                    atomicOr((unsigned long long *)err, (unsigned long long)G5_DEVERR_WAIT);
                    x = 0;
                    break;
                }
            }
            if ((t & 3) == ST_INC) atomicMin(&sh.near_inc, (int)threadIdx.x);
        }
        __syncthreads();
        const int ni = sh.near_inc;
        if ((int)threadIdx.x > ni) x = 0;
        if (__any_sync(0xFFFFFFFFu, x != 0)) {
#pragma unroll
            for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
            if (g5_lane() == 0) atomicAdd(&sh.before, x);
        }
        __syncthreads();
        if (ni < kEB) break;
    }
    __syncthreads();
}

// Word `idx` of a miniblock's payload (word w = idx / 4 of lane l = idx & 3's bit
// stream, ipackwithoutmask<b>, simdintegratedbitpacking.cpp:875) from fields
// of `b` bits at d (field j of lane l at d[4 j + l]): those whose bits j b .. j b
// + b - 1 reach into bits 32 w .. 32 w + 31.
__device__ __forceinline__ uint32_t pack_word(const uint32_t *d, uint32_t b, uint32_t magic, uint32_t idx)
{
    const uint32_t first = 8 * (idx & ~3u), l = idx & 3;  // bit 32 w
    uint32_t j = (first * magic) >> 16;                   // floor(32 w / b)
    int sh = (int)(j * b) - (int)first;                   // at most 0
    uint32_t x = d[4 * j + l] >> -sh;
    for (;;) {
        sh += (int)b;
        ++j;
        if (sh >= 32) break;
        x |= d[4 * j + l] << sh;
    }
    return x;
}

// The payload of a miniblock of width b (1..31) whose deltas are at d, by one
// warp.  Up to 8 bits, a lane first joins four values of a component into one
// field (in place: 32 of them), so that a word gathers at most 32 / 4 b + 2
// fields instead of as many as 32 values.
__device__ __forceinline__ void pack_mb(uint32_t *d, uint32_t b, const uint32_t *magic, uint32_t *dst)
{
    const uint32_t lane = g5_lane();
    uint32_t f = b;
    if (b < 8) {  // (fields of 32 bits would shift by 32)
        const uint32_t *s = d + 16 * (lane >> 2) + (lane & 3);
        const uint32_t x = s[0] | s[4] << b | s[8] << (2 * b) | s[12] << (3 * b);
        __syncwarp();
        d[lane] = x;
        __syncwarp();
        f = 4 * b;
    }
    for (uint32_t i = lane; i < 4 * b; i += 32) dst[i] = pack_word(d, f, magic[f], i);
}

// Chunk c of the queue: its groups to the stream at `out`.  The block with the
// last group also writes the stream header and the tail (in its last warp,
// beside the packing) and leaves the stream's words in *words.
template <bool ANY>
__device__ void enc_chunk(EncShared &sh, const EncLen &e, const uint32_t *in, uint64_t c, uint64_t epoch,
                          unsigned long long *slots, uint32_t stride, uint64_t *err, uint32_t *out, int mode,
                          uint64_t *words)
{
    const int lane = g5_lane(), wid = threadIdx.x >> 5;
    const uint64_t k0 = 16 * c * e.gpc;  // the chunk's first miniblock
    const uint32_t nmb = (uint32_t)min((uint64_t)16 * e.gpc, e.nmb - k0);
    const uint32_t *x = in + 128 * k0;
    // (claim_tile's barriers separate the chunks)
    if (ANY) {
        for (uint32_t p = threadIdx.x; p < 128 * nmb; p += kEB) reinterpret_cast<uint32_t *>(sh.vec)[p] = x[p];
        if (threadIdx.x < 4) reinterpret_cast<uint32_t *>(sh.prev)[threadIdx.x] = k0 ? x[(int)threadIdx.x - 4] : 0u;
    } else {
        const uint4 *v = reinterpret_cast<const uint4 *>(x);
        for (uint32_t p = threadIdx.x; p < 32 * nmb; p += kEB) cp_async16(sh.vec + p, v + p);
        if (threadIdx.x == 0) {
            if (k0) cp_async16(sh.prev, v - 1);
            else sh.prev[0] = make_uint4(0, 0, 0, 0);
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    }
    __syncthreads();
    for (uint32_t m = threadIdx.x + 1; m < nmb; m += kEB) sh.prev[m] = sh.vec[32 * m - 1];
    __syncthreads();
#pragma unroll 2
    for (uint32_t m = wid; m < nmb; m += kEW) {
        uint4 *v = sh.vec + 32 * m;
        const uint4 d = deltas(v[lane], lane ? v[lane - 1] : sh.prev[m], mode);
        const uint32_t b = bits_of(__reduce_or_sync(0xFFFFFFFFu, d.x | d.y | d.z | d.w));
        if (b < 32) v[lane] = d;  // (a raw miniblock keeps its values; the reduction above orders the reads)
        if (lane == 0) sh.b[m] = (uint8_t)b;
    }
    __syncthreads();
    const uint32_t m = threadIdx.x, mb = m < nmb ? sh.b[m] : 0u, head = m < nmb && (m & 15) == 0 ? 4u : 0u;
    uint32_t total;
    const uint32_t at = block_excl_u32(head + 4 * mb, sh.w, total);
    if (m < nmb) sh.off[m] = at + head;
    if (threadIdx.x == 0) put_part(slots + stride * c, total, epoch << 2 | (c ? ST_AGG : ST_INC));
    enc_before(sh, c, epoch, slots, stride, err);
    const uint64_t base = 4 + sh.before;  // word of the chunk's first header
    if (c && e.nchunks > (uint64_t)kEB && threadIdx.x == 0)
        put_part(slots + stride * c, sh.before + total, epoch << 2 | ST_INC);
    uint32_t *o = out + base;
    // the 16 widths of each group, big-endian bytes in each word; 0 where a last
    // group has no miniblock (simdbinarypacking.h:200-214)
    const uint32_t groups = (nmb + 15) / 16;
    if (threadIdx.x < 4 * groups) {
        const uint32_t g = threadIdx.x / 4, k = threadIdx.x & 3;
        uint32_t hw = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t i = 16 * g + 4 * k + q;
            hw |= (i < nmb ? sh.b[i] : 0u) << (24 - 8 * q);
        }
        o[sh.off[16 * g] - 4 + k] = hw;
    }
    uint32_t warps = kEW;
    if (c + 1 == e.nchunks) {
        --warps;
        if (wid == (int)warps) {
            const uint64_t w = enc_tail_warp(in, e.n, e.n1, base + total, out, sh.bytes);
            if (lane == 0) *words = w;
            return;
        }
    }
    for (uint32_t q = wid; q < nmb; q += warps) {
        const uint32_t b = sh.b[q];
        uint32_t *dst = o + sh.off[q];
        if (b == 32) reinterpret_cast<uint4 *>(dst)[lane] = sh.vec[32 * q + lane];
        else if (b) pack_mb(reinterpret_cast<uint32_t *>(sh.vec + 32 * q), b, sh.magic, dst);
    }
}

__global__ void __launch_bounds__(kEB, 3) k_encode(const uint32_t *__restrict__ in, const uint64_t *n_dev, uint64_t n_val,
                                                uint64_t max_n, uint64_t raw_thr, uint32_t *__restrict__ out,
                                                uint64_t *scal, unsigned long long *slots, uint32_t stride,
                                                uint64_t *words_out, uint64_t *result, int mode)
{
    extern __shared__ __align__(16) unsigned char s_dyn_e[];
    EncShared &sh = *reinterpret_cast<EncShared *>(s_dyn_e);
    if (threadIdx.x >= 1 && threadIdx.x < 32) sh.magic[threadIdx.x] = 65536u / threadIdx.x + 1u;
    g5_pdl_sync();
    const uint64_t epoch = scal[CS_E_EPOCH];
    const EncLen e = enc_len(n_dev ? *n_dev : n_val, max_n, raw_thr, gridDim.x);
    // a queue of one chunk is block 0's alone: no claim and no counting out
    // (3000 ids there and back through the plugin 55.2 -> 52.7 us, a scale-22
    // search with the codec 436 -> 428).  Not where the words go to the place of
    // the length: a block that starts late would read them as one
    const bool lone = (!n_dev || n_dev != words_out) && (e.raw ? e.n <= kLoneRaw : e.nchunks <= 1);
    if (lone && blockIdx.x) return;
    if (e.raw) {
        const uint64_t step = lone ? kEB : (uint64_t)gridDim.x * kEB;
        for (uint64_t i = (uint64_t)blockIdx.x * kEB + threadIdx.x; i < e.n; i += step) out[i] = in[i];
    } else if (!e.too_long) {
        for (;;) {
            const uint64_t c = lone ? 0 : claim_tile(&scal[CS_E_CTR], &sh.t);
            if (c >= e.nchunks) break;
            enc_chunk<false>(sh, e, in, c, epoch, slots, stride, &scal[CS_E_ERR], out, mode, &scal[CS_E_WORDS]);
            // every block has drawn one: none is left (5 M values 26.4 -> 25.5 us a call)
            if (e.nchunks <= gridDim.x) break;
        }
        if (e.ng == 0 && blockIdx.x == 0 && threadIdx.x < 32) {
            const uint64_t w = enc_tail_warp(in, e.n, 0, 4, out, sh.bytes);
            if (threadIdx.x == 0) scal[CS_E_WORDS] = w;
        }
    }
    if (lone) __syncthreads();
    if (lone ? threadIdx.x == 0 : last_block(&scal[CS_E_DONE])) {
        __threadfence();
        uint64_t err = vload64(&scal[CS_E_ERR]);
        if (e.too_long) err |= G5_DEVERR_CAPACITY;
        const uint64_t w = e.raw ? e.n : e.too_long ? 0 : vload64(&scal[CS_E_WORDS]);
        scal[CS_N] = e.n;
        scal[CS_N1] = e.n1;
        scal[CS_ERR] = err;
        if (!e.too_long) {
            scal[CS_WORDS] = w;
            if (words_out) *words_out = w;
        }
        if (result) {
            result[0] = e.n;
            result[1] = w;
            result[2] = err;
        }
        scal[CS_E_CTR] = 0;
        scal[CS_E_DONE] = 0;
        scal[CS_E_ERR] = 0;
        scal[CS_E_EPOCH] = epoch + 1;
        __threadfence();
    }
}

// ---- decoder ---------------------------------------------------------------------------
//
// One launch.  A group's position is only given by the chain of group headers
// before it (each says how long its group is), and its values need the sums of
// all groups before it.  The stream's vectors are cut into chunks, a block per
// chunk, its groups (the ones that start in it) decoded from shared memory:
//
//   entry   where the chain enters the chunk.  The group before the entry
//           starts at most kSpan vectors before the chunk; the block tries every
//           vector there that could be a header (16 bytes of at most 32: payload
//           hardly ever is) and follows the chain from where it leads.  Where
//           exactly one entry comes up whose chain reaches the next chunk, that
//           is the one, known without any other chunk.  The first chunk's entry
//           is given.  (Near the stream's end the chain may stop in the chunk:
//           there every entry counts.)  Else the block waits for the chunk before
//           to tell its exit, which that one mostly knows all the same: chains
//           from several entries run together.  (Only miniblocks of a bit or
//           two look like headers; no sorted queue of distinct ids has them.)
//   sums    the lane sums of every miniblock and, in order, of the chunk
//           (a raw b = 32 miniblock restarts them)
//   meet    the chunk publishes its entry, exit, groups and sums, and adds up
//           those of all chunks before it: 512 of them are read at once, so on
//           streams up to a wave there is one round trip and no chain.  Each
//           chunk checks its entry against the exit before it; a chain that
//           breaks before the last group makes the stream corrupt.
//   values  the miniblocks are unpacked again, now with their base
//
// What bounds it: a chain of round trips whatever the size (ticket and stream
// header 1.2 us, chunk 0.6, candidates 0.9, groups 0.6, sums 1.5-2.4, meeting
// 1.2-3, the last block's exit 1) and, on large streams, the values (5 us for 20
// MB: issue and the stores).  5 M values of 6 bits take 17 us, against 50 us for
// the four launches this replaced (transfer tables from every entry, a
// one-block walk through them, positions, an unpacker with a look-back chain
// over its tiles); 3000 values 7 us against 12.  Unpacking twice is cheaper
// than keeping a chunk's values (128 KB at 6 bits) in shared memory, which
// would leave one block per SM.
constexpr int kSpan = 513;         // a group spans at most 1 + 16 * 32 vectors
constexpr uint32_t kDead = 0xFFFFu;
constexpr int kDB = 512;           // threads per block
constexpr int kDW = kDB / 32;
constexpr uint32_t kMinChunk = 16, kMidChunk = 576, kMaxChunk = 1536;  // vectors per chunk
constexpr uint64_t kChunkValues = 32768;  // values a chunk shorter than kMidChunk should have
constexpr int kDG = 32;            // groups whose miniblocks are held together
constexpr int kDM = 16 * kDG;

// What a chunk tells the ones after it: the groups it starts and their sums
// (ST_AGG), or those of all chunks up to it (ST_INC): three parts of one status.
struct ChunkRec {
    uint4 v;
    uint32_t f;       // the sums restart in the chunk
    uint32_t exit;    // where the chain enters the next chunk (kDead: it does not)
    uint32_t groups;
};
// The fourth part is the exit alone, published before the sums, so that a run
// of chunks that wait for their entries waits for a walk each and no more.
struct __align__(128) ChunkSlot {  // (a line each: all blocks read all of them at once)
    unsigned long long part[4][2];
};

struct DecShared {
    uint4 vec[kMaxChunk + kSpan + 1];  // the chunk, the rest of its last group, one more read by unpack4
    uint16_t jump[kMaxChunk];             // where the group at a vector ends, if it is a header
    uint16_t gpos[kMaxChunk];             // the chunk's groups
    uint32_t mb[kDM];                     // miniblocks: payload vector | width << 16
    uint4 v[kDM];                         // their sums, then the sums before them
    uint8_t f[kDM];
    uint32_t tail[kTailMaxBytes / 4];
    uint4 wv[kDW];                        // warp totals of a scan
    uint32_t wf[kDW];
    uint64_t t;
    uint32_t entry, exit, groups;
    uint32_t stop;                        // the vector the chain stops at, if it is in the chunk
    uint32_t first, last;                 // least and greatest entry that came up
    uint32_t xfirst, xlast;               // and exit their chains lead to
    uint4 cv;                             // the chunk's sums
    uint32_t cf;
    unsigned long long before;            // groups before the chunk
    uint4 base;                           // sums before the chunk
    int near_reset, near_inc;             // nearest record before that restarts the sums / holds them all
};

__device__ __forceinline__ uint4 add4(uint4 a, uint4 b)
{
    return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// Header checks every block makes alike.
struct DecHead {
    uint64_t words, nv, n1, nmb, ng, nchunks;
    uint32_t S;  // vectors per chunk
    bool raw, bad;
};

// Chunk size of a stream of nv vectors and n1 values in whole miniblocks, `per`
// vectors a block's share: that, but no chunk shorter than kMidChunk unless the
// stream packs so many values into a vector that such chunks would hold far
// more than kChunkValues.
__host__ __device__ __forceinline__ uint32_t dec_chunk_size(uint64_t nv, uint64_t n1, uint64_t per)
{
    uint64_t few = kMidChunk;
    if (n1 > kChunkValues && kChunkValues * nv / n1 < few) few = kChunkValues * nv / n1;
    const uint64_t s = ((per > few ? per : few) + kMinChunk - 1) / kMinChunk * kMinChunk;
    return s < kMinChunk ? kMinChunk : s > kMaxChunk ? kMaxChunk : (uint32_t)s;
}

__device__ __forceinline__ DecHead dec_head(const uint32_t *in, uint64_t words, uint64_t cap, uint64_t raw_thr,
                                            const uint64_t *n_expect, uint64_t max_vec, uint64_t max_mb,
                                            uint32_t blocks)
{
    DecHead h;
    h.words = words;
    h.nv = words / 4;
    h.n1 = h.nmb = h.ng = h.nchunks = 0;
    h.S = kMidChunk;
    h.bad = false;
    // plugin semantics: raw when n <= thr or the stream is as long as n
    // (cpu_2d/compression/cpusimd.hh:169-173)
    h.raw = raw_thr && n_expect && (*n_expect <= raw_thr || words == *n_expect);
    if (h.raw) {
        h.bad = words > cap;
        return h;
    }
    if (words < 4) {
        h.bad = true;
    } else {
        const uint4 x = *reinterpret_cast<const uint4 *>(in);
        h.n1 = x.x;
        if (x.y != kCookie || x.z != kCookie || x.w != kCookie) h.bad = true;
        if (h.n1 % 128 || h.n1 > cap || h.n1 / 128 >= max_mb) h.bad = true;
        // groups but no vector that could hold one's header: there is no chunk
        // that would find the chain broken
        if (h.n1 && h.nv < 2) h.bad = true;
    }
    if (h.nv > max_vec) h.bad = true;
    if (h.bad) h.n1 = 0;
    h.nmb = h.n1 / 128;
    h.ng = (h.nmb + 15) / 16;
    if (!h.bad) h.S = dec_chunk_size(h.nv, h.n1, (h.nv + blocks - 1) / blocks);
    h.nchunks = h.ng ? (h.nv - 1 + h.S - 1) / h.S : 0;
    return h;
}

__device__ __forceinline__ uint32_t width_of(uint4 h, int i)
{
    const uint32_t w = i < 4 ? h.x : i < 8 ? h.y : i < 12 ? h.z : h.w;
    return (w >> (24 - 8 * (i & 3))) & 0xFFu;
}

// Sum of the 16 widths (bytes) of a vector taken as a group header, or kDead
// if one is above 32.
__device__ __forceinline__ uint32_t header_sum(uint4 x)
{
    const uint32_t over = __vcmpgtu4(x.x, 0x20202020u) | __vcmpgtu4(x.y, 0x20202020u) |
                          __vcmpgtu4(x.z, 0x20202020u) | __vcmpgtu4(x.w, 0x20202020u);
    uint32_t sum = __dp4a(x.x, 0x01010101u, 0u);
    sum = __dp4a(x.y, 0x01010101u, sum);
    sum = __dp4a(x.z, 0x01010101u, sum);
    sum = __dp4a(x.w, 0x01010101u, sum);
    return over ? kDead : sum;
}

// Sum of the first i widths of a group header (its leading, big-endian bytes).
__device__ __forceinline__ uint32_t header_before(uint4 h, int i)
{
    const uint32_t x[4] = {h.x, h.y, h.z, h.w};
    uint32_t sum = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int keep = i - 4 * j;
        const uint32_t m = keep >= 4 ? 0xFFFFFFFFu : keep <= 0 ? 0u : ~(0xFFFFFFFFu >> (8 * keep));
        sum = __dp4a(x[j] & m, 0x01010101u, sum);
    }
    return sum;
}

// Values 4 q .. 4 q + 3 of component l of a miniblock (l = lane & 3, q = lane >> 2)
// whose payload starts at word s and has width b.
__device__ __forceinline__ void unpack4(const uint32_t *s, uint32_t b, uint32_t (&v)[4])
{
    const uint32_t l = g5_lane() & 3, q = g5_lane() >> 2;
    if (b == 32) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = s[16 * q + 4 * i + l];
        return;
    }
    const uint32_t mask = (1u << b) - 1u;
    uint32_t bit = 4 * q * b;
#pragma unroll
    for (int i = 0; i < 4; ++i, bit += b) {
        const uint32_t *p = s + 4 * (bit >> 5) + l;
        v[i] = __funnelshift_r(p[0], p[4], bit) & mask;
    }
}

// The sum of component l of a miniblock whose payload starts at word s, by one
// thread: d4 adds each component; dm adds component 3 (every component of a
// vector is relative to component 3 of the vector before); a raw miniblock
// gives its last vector.  A thread walking its 32 values costs a third of the
// issue slots of a warp unpacking them and adding them up by shuffles.
__device__ __forceinline__ uint32_t mb_sum(const uint32_t *s, uint32_t b, uint32_t l)
{
    if (b == 32) return s[124 + l];
    const uint32_t mask = (1u << b) - 1u;
    uint32_t w0 = s[l], w1 = s[4 + l], bit = 0, sum = 0;
    const uint32_t *p = s + 8 + l;
#pragma unroll 8
    for (int j = 0; j < 32; ++j) {
        sum += __funnelshift_r(w0, w1, bit) & mask;
        bit += b;
        if (bit >= 32) {
            bit -= 32;
            w0 = w1;
            w1 = *p;
            p += 4;
        }
    }
    return sum;
}

// Lane j's vector j of a miniblock with the sums `base` before it.
__device__ __forceinline__ uint4 mb_values(const uint32_t *s, uint32_t b, uint4 base, int mode)
{
    const int lane = g5_lane(), l = lane & 3;
    if (b == 32) return reinterpret_cast<const uint4 *>(s)[lane];
    uint32_t v[4];
    unpack4(s, b, v);
    // running sums of the lane's four values, then of the eight lanes of its
    // component
    uint32_t p[4];
    p[0] = v[0];
    p[1] = p[0] + v[1];
    p[2] = p[1] + v[2];
    p[3] = p[2] + v[3];
    uint32_t inc = p[3];
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += y;
    }
    const uint32_t ex = inc - p[3];
    if (mode == G5_CODEC_DM) {
        // components 0..2 add component 3 of the vector before
        const uint32_t c = base.w + ex;
        const int w = lane | 3;
        uint32_t before[4];
        before[0] = __shfl_sync(0xFFFFFFFFu, c, w);
#pragma unroll
        for (int i = 0; i < 3; ++i) before[i + 1] = __shfl_sync(0xFFFFFFFFu, c + p[i], w);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = l == 3 ? c + p[i] : before[i] + v[i];
    } else {
        const uint32_t c = ex + (l == 0 ? base.x : l == 1 ? base.y : l == 2 ? base.z : base.w);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = c + p[i];
    }
    // the four lanes of a q hold vectors 4 q .. 4 q + 3 by component: transposed,
    // each holds one vector
    uint32_t a = __shfl_xor_sync(0xFFFFFFFFu, l & 1 ? v[0] : v[1], 1), c = __shfl_xor_sync(0xFFFFFFFFu, l & 1 ? v[2] : v[3], 1);
    if (l & 1) {
        v[0] = a;
        v[2] = c;
    } else {
        v[1] = a;
        v[3] = c;
    }
    a = __shfl_xor_sync(0xFFFFFFFFu, l & 2 ? v[0] : v[2], 2);
    c = __shfl_xor_sync(0xFFFFFFFFu, l & 2 ? v[1] : v[3], 2);
    if (l & 2) {
        v[0] = a;
        v[1] = c;
    } else {
        v[2] = a;
        v[3] = c;
    }
    return make_uint4(v[0], v[1], v[2], v[3]);
}

// Publishes a chunk's record (three threads of a warp, a part each).
__device__ __forceinline__ void publish(ChunkSlot *p, const ChunkRec &r, uint64_t epoch, uint32_t flag)
{
    const int k = g5_lane();
    if (k < 3)
        put_part(p->part[k],
                 k == 0   ? r.v.x | (unsigned long long)r.v.y << 32
                 : k == 1 ? r.v.z | (unsigned long long)r.v.w << 32
                          : r.groups | (unsigned long long)r.exit << 32 | (unsigned long long)r.f << 63,
                 epoch << 2 | flag);
}

// Waits for a chunk's exit; kDead past the limit.
__device__ __forceinline__ uint32_t await_exit(const ChunkSlot *p, uint64_t epoch, uint64_t *err)
{
    for (uint32_t spins = 0; spins <= kSpinLimit; ++spins) {
        unsigned long long x, t;
        get_part(p->part[3], x, t);
        if ((t >> 2) == epoch) return (uint32_t)x;
    }
    atomicOr((unsigned long long *)err, (unsigned long long)G5_DEVERR_WAIT);
    return kDead;
}

// Waits for a chunk's record; its flag, or ST_NONE past the limit.
__device__ __forceinline__ uint32_t await_record(const ChunkSlot *p, uint64_t epoch, ChunkRec &r)
{
    for (uint32_t spins = 0; spins <= kSpinLimit; ++spins) {
        unsigned long long x[3], t[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) get_part(p->part[k], x[k], t[k]);
        if ((t[0] >> 2) == epoch && t[0] == t[1] && t[0] == t[2]) {
            r.v = make_uint4((uint32_t)x[0], (uint32_t)(x[0] >> 32), (uint32_t)x[1], (uint32_t)(x[1] >> 32));
            r.groups = (uint32_t)x[2];
            r.exit = (uint32_t)(x[2] >> 32) & 0x7FFFFFFFu;
            r.f = (uint32_t)(x[2] >> 63);
            return (uint32_t)(t[0] & 3u);
        }
    }
    return ST_NONE;
}

// The groups and sums of chunks 0 .. c - 1, by the whole block, into sh.before
// and sh.base; sh.exit: where the chain leaves chunk c - 1.  The stream's
// records start at slots.
__device__ void dec_before(DecShared &sh, uint64_t c, uint64_t epoch, const ChunkSlot *slots, uint64_t *err)
{
    if (threadIdx.x == 0) {
        sh.before = 0;
        sh.base = make_uint4(0, 0, 0, 0);
    }
    bool sums = true;  // no restart met yet
    for (int64_t hi = (int64_t)c - 1; hi >= 0; hi -= kDB) {
        if (threadIdx.x == 0) sh.near_reset = sh.near_inc = kDB;
        __syncthreads();
        const int64_t j = hi - threadIdx.x;  // thread 0: the nearest
        ChunkRec r;
        r.v = make_uint4(0, 0, 0, 0);
        r.f = r.groups = 0;
        r.exit = kDead;
        if (j >= 0) {
            const uint32_t flag = await_record(slots + j, epoch, r);
            if (flag == ST_NONE) atomicOr((unsigned long long *)err, (unsigned long long)G5_DEVERR_WAIT);
            const bool all = flag == ST_INC;
            if (all) atomicMin(&sh.near_inc, (int)threadIdx.x);
            if (all || r.f) atomicMin(&sh.near_reset, (int)threadIdx.x);
            if (hi == (int64_t)c - 1 && threadIdx.x == 0) sh.exit = r.exit;
        }
        __syncthreads();
        const int ni = sh.near_inc, nr = sh.near_reset;
        uint32_t g = (int)threadIdx.x <= ni ? r.groups : 0u;
        uint4 v = sums && (int)threadIdx.x <= nr ? r.v : make_uint4(0, 0, 0, 0);
        if (__any_sync(0xFFFFFFFFu, j >= 0)) {
            g = __reduce_add_sync(0xFFFFFFFFu, g);
            v.x = __reduce_add_sync(0xFFFFFFFFu, v.x);
            v.y = __reduce_add_sync(0xFFFFFFFFu, v.y);
            v.z = __reduce_add_sync(0xFFFFFFFFu, v.z);
            v.w = __reduce_add_sync(0xFFFFFFFFu, v.w);
            if (g5_lane() == 0) {
                atomicAdd(&sh.before, (unsigned long long)g);
                atomicAdd(&sh.base.x, v.x);
                atomicAdd(&sh.base.y, v.y);
                atomicAdd(&sh.base.z, v.z);
                atomicAdd(&sh.base.w, v.w);
            }
        }
        __syncthreads();
        sums = sums && nr == kDB;
        if (ni < kDB) break;
    }
    __syncthreads();
}

// Groups g0 .. g0 + cnt - 1 of the chunk (cnt <= kDG): their miniblocks' places
// and widths (the first `nmb` of them), sums, and the sums before each from
// the first on, `carry` before that; the total comes back in carry.
__device__ void dec_sums(DecShared &sh, uint32_t g0, uint32_t nmb, int mode, uint4 &carry, uint32_t &carry_f)
{
    const int lane = g5_lane(), wid = threadIdx.x >> 5;
    const uint32_t m = threadIdx.x;
    __syncthreads();
    if (m < nmb) {
        const uint32_t p = sh.gpos[g0 + m / 16];
        const uint4 h = sh.vec[p];
        sh.mb[m] = (p + 1 + header_before(h, m & 15)) | width_of(h, m & 15) << 16;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < 4 * nmb; k += kDB) {
        const uint32_t x = sh.mb[k / 4], b = x >> 16;
        const bool dm = mode == G5_CODEC_DM && b != 32;
        reinterpret_cast<uint32_t *>(sh.v)[k] =
            mb_sum(reinterpret_cast<const uint32_t *>(sh.vec + (x & 0xFFFFu)), b, dm ? 3 : k & 3);
        if ((k & 3) == 0) sh.f[k / 4] = b == 32;
    }
    __syncthreads();
    // exclusive scan with restarts over the miniblocks, one per thread
    VecFlag x = ResetAdd::id();
    if (m < nmb) {
        x.v = sh.v[m];
        x.f = sh.f[m];
    }
    const uint32_t warps = (nmb + 31) / 32;
    VecFlag inc = x;
    if ((uint32_t)wid < warps) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const VecFlag y = ResetAdd::shfl_up(inc, o);
            if (lane >= o) inc = ResetAdd::op(y, inc);
        }
        if (lane == 31) {
            sh.wv[wid] = inc.v;
            sh.wf[wid] = inc.f;
        }
    }
    __syncthreads();
    VecFlag pre;
    pre.v = carry;
    pre.f = carry_f;
    VecFlag mine = pre;
    for (uint32_t w = 0; w < warps; ++w) {
        VecFlag t;
        t.v = sh.wv[w];
        t.f = sh.wf[w];
        if (w == (uint32_t)wid) mine = pre;
        pre = ResetAdd::op(pre, t);
    }
    carry = pre.v;
    carry_f = pre.f;
    if ((uint32_t)wid < warps) {
        VecFlag ex = ResetAdd::shfl_up(inc, 1);
        if (lane == 0) ex = ResetAdd::id();
        ex = ResetAdd::op(mine, ex);
        if (m < nmb) {
            sh.v[m] = ex.v;
            // bit 1: the miniblock's base does not include what is before the chunk
            sh.f[m] = (uint8_t)(x.f | (ex.f ? 2u : 0u));
        }
    }
    __syncthreads();
}

// VariableByte tail decoded by one warp (variablebyte.h:217-): nbytes bytes
// in bb (shared memory), values from out[o] on, each the running sum of the
// decoded deltas from 0; o (warp-uniform) ends past the last value.  A byte
// with the high bit ends a value; a sixth byte of one value (a fifth byte
// without the high bit) or an output index at cap makes the stream corrupt
// and ends the decode there, as the sequential decoder does.  32 bytes per
// round: a ballot marks the values' last bytes, the lane holding one
// gathers its value's bytes from the previous last byte on, and a warp scan
// of the values gives the running sums.
__device__ void dec_tail_warp(const uint8_t *bb, uint32_t nbytes, uint64_t cap, uint32_t *out,
                              const uint32_t *expect, uint64_t &o, uint64_t &e)
{
    const int lane = g5_lane();
    const unsigned lt = g5_lanemask_lt();
    uint32_t run = 0;    // the last value so far
    int last_end = -1;   // byte index of the last value's last byte
    for (uint32_t b0 = 0; b0 < nbytes; b0 += 32) {
        const uint32_t pb = b0 + lane;
        const bool in_range = pb < nbytes;
        const bool term = in_range && (bb[pb] & 128u);
        const unsigned tm = __ballot_sync(0xFFFFFFFFu, term);
        const unsigned below = tm & lt;
        const int prev_end = below ? (int)(b0 + 31 - __clz(below)) : last_end;
        // the fifth byte of a value without the high bit
        const unsigned em = __ballot_sync(0xFFFFFFFFu, in_range && !term && (int)pb - prev_end >= 5);
        unsigned ok = em ? tm & ((1u << (__ffs(em) - 1)) - 1u) : tm;  // values ending before it
        // output capacity, checked value by value
        const uint64_t room = cap > o ? cap - o : 0;
        if ((uint64_t)__popc(ok) > room) {
            unsigned keep = ok;
            for (uint64_t k = 0; k < room; ++k) keep &= keep - 1;  // drop the first `room` values
            ok &= ~keep;
            e |= G5_DEVERR_CORRUPT;
        }
        if (em) e |= G5_DEVERR_CORRUPT;
        const bool mine = (ok >> lane) & 1u;
        uint32_t v = 0;
        if (mine)
            for (int k = prev_end + 1, sh = 0; k <= (int)pb; ++k, sh += 7) v |= (uint32_t)(bb[k] & 127u) << sh;
        uint32_t inc = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
            if (lane >= d) inc += y;
        }
        if (mine) {
            const uint64_t idx = o + __popc(ok & lt);
            const uint32_t val = run + inc;
            out[idx] = val;
            if (expect && expect[idx] != val) e |= G5_DEVERR_MISMATCH;
        }
        o += __popc(ok);
        run += __shfl_sync(0xFFFFFFFFu, inc, 31);
        if (tm) last_end = (int)(b0 + 31 - __clz(tm));
        if (e & G5_DEVERR_CORRUPT) break;
    }
    // the lanes' mismatch flags into one
    e |= __reduce_or_sync(0xFFFFFFFFu, (unsigned)(e & G5_DEVERR_MISMATCH)) ? G5_DEVERR_MISMATCH : 0;
}

// Lane j's vector j of miniblock k held in sh (dec_sums).
__device__ __forceinline__ uint4 held_values(const DecShared &sh, uint32_t k, int mode)
{
    const uint32_t x = sh.mb[k];
    uint4 base = sh.v[k];
    if (!(sh.f[k] & 2)) base = add4(base, sh.base);
    return mb_values(reinterpret_cast<const uint32_t *>(sh.vec + (x & 0xFFFFu)), x >> 16, base, mode);
}

// Writes them, to out (miniblock 0's values first); true if one differs from
// `expect`.  ANY: out has no alignment.
template <bool ANY>
__device__ __forceinline__ bool put_values(uint4 v, uint32_t k, uint32_t *out, const uint32_t *expect)
{
    const uint64_t at = 32 * (uint64_t)k + g5_lane();
    if (ANY) {
        uint32_t *o = out + 4 * at;
        o[0] = v.x;
        o[1] = v.y;
        o[2] = v.z;
        o[3] = v.w;
        return false;
    }
    reinterpret_cast<uint4 *>(out)[at] = v;
    if (!expect) return false;
    const uint4 e = reinterpret_cast<const uint4 *>(expect)[at];
    return (e.x != v.x) | (e.y != v.y) | (e.z != v.z) | (e.w != v.w);
}

// The values of miniblocks 0 .. nmb - 1 held in sh, by warps 0 .. warps - 1 two
// at a time (one miniblock's chain of shuffles leaves the issue slots half
// empty).
template <bool ANY>
__device__ __forceinline__ bool dec_out(DecShared &sh, uint32_t nmb, uint32_t warps, uint32_t *out,
                                        const uint32_t *expect, int mode)
{
    bool bad = false;
    uint32_t k = threadIdx.x >> 5;
    if (k >= warps) return false;
    for (; k + warps < nmb; k += 2 * warps) {
        const uint4 v = held_values(sh, k, mode), u = held_values(sh, k + warps, mode);
        bad |= put_values<ANY>(v, k, out, expect);
        bad |= put_values<ANY>(u, k + warps, out, expect);
    }
    if (k < nmb) bad |= put_values<ANY>(held_values(sh, k, mode), k, out, expect);
    return bad;
}

// The VariableByte tail of a stream (variablebyte.h:217-), words from blkend
// on, by one warp: values to out[n1 ..], their end in n.  Returns error bits.
__device__ __noinline__ uint32_t dec_tail(uint32_t *s_b, const uint32_t *in, uint64_t words, uint64_t blkend,
                                          uint64_t n1, uint64_t cap, uint32_t *out, const uint32_t *expect, uint64_t &n)
{
    const uint64_t tw = words > blkend ? words - blkend : 0;
    n = 0;
    if (tw * 4 > kTailMaxBytes) return G5_DEVERR_CORRUPT;
    for (uint64_t i = g5_lane(); i < tw; i += 32) s_b[i] = in[blkend + i];
    __syncwarp();
    uint64_t o = n1, e = 0;
    dec_tail_warp(reinterpret_cast<const uint8_t *>(s_b), (uint32_t)(tw * 4), cap, out, expect, o, e);
    n = o;
    return (uint32_t)e;
}

// Chunk c of the stream `in`: decodes the groups that start in it.  Returns
// error bits (of this thread).  The block whose chunk holds the last group also
// decodes the tail (in its last warp, beside the values) and leaves the
// stream's value count in *count.
template <bool ANY>
__device__ uint32_t dec_chunk(DecShared &sh, const DecHead &h, const uint32_t *in, uint64_t c, uint64_t epoch,
                              ChunkSlot *slots, uint64_t *err, uint32_t *out, uint64_t cap, const uint32_t *expect,
                              int mode, uint64_t *count)
{
    const uint32_t S = h.S;
    const uint64_t a = 1 + c * S;  // the chunk's first vector
    const uint32_t len = (uint32_t)min((uint64_t)S, h.nv - a), have = (uint32_t)min((uint64_t)S + kSpan, h.nv - a);
    const uint4 *v = reinterpret_cast<const uint4 *>(in) + a, *before = v - kSpan;
    __syncthreads();  // the chunk before is no longer read
    for (uint32_t p = threadIdx.x; p < have; p += kDB) cp_async16(sh.vec + p, v + p);
    if (threadIdx.x == 0) {
        sh.vec[have] = make_uint4(0, 0, 0, 0);
        sh.first = sh.xfirst = kDead;
        sh.last = sh.xlast = 0;
        sh.entry = c == 0 ? 0u : kDead;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    for (uint32_t p = threadIdx.x; p < len; p += kDB) {
        const uint32_t sum = header_sum(sh.vec[p]);
        sh.jump[p] = (uint16_t)(sum != kDead && a + p + 1 + sum <= h.nv ? p + 1 + sum : kDead);
    }
    __syncthreads();
    // far enough from the end that a block part ending in this chunk would
    // leave more tail than any stream has (kTailMaxBytes)
    const bool inner = a + S + kSpan + kTailMaxBytes / 16 + 1 <= h.nv;
    if (c > 0) {
        for (uint32_t k = threadIdx.x; k < kSpan; k += kDB) {
            if (a + k < kSpan + 1) continue;  // (before the first group)
            const uint32_t sum = header_sum(before[k]);  // kSpan - k vectors before the chunk
            if (sum == kDead || k + 1 + sum < kSpan) continue;
            const uint32_t e = k + 1 + sum - kSpan;
            uint32_t p = e;
            while (inner && p < S) p = sh.jump[p];  // (kDead is past S)
            if (p != kDead) {
                atomicMin(&sh.first, e);
                atomicMax(&sh.last, e);
                atomicMin(&sh.xfirst, p - S);
                atomicMax(&sh.xlast, p - S);
            }
        }
        __syncthreads();
    }
    // the chunk's groups: down the chain to the chunk's end or to a vector that
    // is no header (no vector of a tail is: each value ends in a byte above 127)
    if (threadIdx.x == 0) {
        if (c > 0 && sh.first != kDead && sh.first == sh.last) {
            sh.entry = sh.first;
        } else if (c > 0) {
            // (one of the entries that came up is the real one)
            if (inner && sh.first != kDead && sh.xfirst == sh.xlast)
                put_part(slots[c].part[3], sh.xfirst, epoch << 2 | ST_AGG);
            sh.entry = await_exit(slots + c - 1, epoch, err);
        }
        uint32_t p = sh.entry, g = 0, nx = p;
        while (p < len && (nx = sh.jump[p]) != kDead) {
            sh.gpos[g++] = (uint16_t)p;
            p = nx;
        }
        sh.groups = g;
        sh.exit = nx == kDead || len < S ? kDead : p - S;
        sh.stop = nx == kDead && p < len ? p : kDead;
        put_part(slots[c].part[3], sh.exit, epoch << 2 | ST_AGG);
    }
    __syncthreads();
    uint32_t groups = sh.groups;
    const uint32_t exit = sh.exit, entry = sh.entry;
    // sums of the whole chunk (a last group that is not full has widths of 0
    // where its miniblocks are missing: they add nothing)
    uint4 cv = make_uint4(0, 0, 0, 0);
    uint32_t cf = 0;
    const uint32_t batches = (groups + kDG - 1) / kDG;
    for (uint32_t i = 0; i < batches; ++i)
        dec_sums(sh, i * kDG, min(16 * (groups - i * kDG), (uint32_t)kDM), mode, cv, cf);
    // publish, then add up what is before (the first chunk's own sums are all
    // there are up to it)
    ChunkRec r;
    r.v = cv;
    r.f = cf;
    r.exit = exit;
    r.groups = groups;
    if (threadIdx.x < 32) publish(slots + c, r, epoch, c == 0 ? ST_INC : ST_AGG);
    dec_before(sh, c, epoch, slots, err);
    if (c > 0) {
        if (h.nchunks > (uint64_t)kDB && threadIdx.x < 32) {
            // more chunks than one look reaches: everything up to this one
            r.v = cf ? cv : add4(cv, sh.base);
            r.f = 1;
            r.groups = (uint32_t)(sh.before + groups);
            publish(slots + c, r, epoch, ST_INC);
        }
        if (sh.before < h.ng && sh.exit != kDead && sh.exit != entry) return G5_DEVERR_CORRUPT;
    }
    const bool ended = c > 0 && sh.exit == kDead;
    const uint64_t first = sh.before;
    // the chain ended before this chunk (there it was checked to be complete)
    if (first >= h.ng || ended) return 0;
    const uint32_t rest = (uint32_t)(h.nmb - 16 * (h.ng - 1));  // miniblocks of the last group
    bool again = batches > 1;  // the sums held are not the first batch's
    if (first + groups < h.ng && sh.stop != kDead) {
        // the chain stops before the last group, unless this is the last one,
        // whose header need not be one past its `rest` widths
        const uint32_t p = sh.stop;
        const uint4 hv = sh.vec[p];
        bool ok = first + groups + 1 == h.ng && a + p + 1 + header_before(hv, (int)rest) <= h.nv;
        for (uint32_t q = 0; q < rest; ++q) ok &= width_of(hv, (int)q) <= 32;
        if (!ok) return G5_DEVERR_CORRUPT;
        if (threadIdx.x == 0) sh.gpos[groups] = (uint16_t)p;
        ++groups;
        again = true;  // (dec_sums begins with a barrier)
    }
    const uint32_t nmb = (uint32_t)min((uint64_t)16 * groups, h.nmb - 16 * first);
    uint32_t bad = 0, warps = kDW;
    if (first + groups >= h.ng) {
        // the stream's last group, which may hold fewer miniblocks
        if (again) __syncthreads();
        --warps;
        if (threadIdx.x >> 5 == warps) {
            const uint32_t p = sh.gpos[h.ng - 1 - first];
            uint64_t n;
            bad = dec_tail(sh.tail, in, h.words, 4 * (a + p + 1 + header_before(sh.vec[p], (int)rest)), h.n1, cap, out,
                           expect, n);
            if (g5_lane() == 0) *count = n;
        }
    } else if (c + 1 == h.nchunks) {
        return G5_DEVERR_CORRUPT;  // the stream ends before the last group
    }
    const uint64_t k0 = 16 * first;
    bool diff = false;
    uint4 rv = make_uint4(0, 0, 0, 0);
    uint32_t rf = 0;
    for (uint32_t i = 0; i * kDM < nmb; ++i) {
        const uint32_t n = min(nmb - i * kDM, (uint32_t)kDM);
        if (again) dec_sums(sh, i * kDG, n, mode, rv, rf);
        const uint64_t at = 128 * (k0 + (uint64_t)i * kDM);
        diff |= dec_out<ANY>(sh, n, warps, out + at, expect ? expect + at : nullptr, mode);
    }
    return bad | (diff ? (uint32_t)G5_DEVERR_MISMATCH : 0u);
}

// One stream.  With `expect` every value is compared with the expected one
// (the level loop's round-trip check); `acc` accumulates words and values; the
// count goes to n_out and, with the words and error bits, to `result` (pinned
// host memory), each if given.  Blocks claim chunks in launch order, so a
// chunk only ever waits on chunks whose blocks already run; records hold the
// call's epoch, so what earlier calls left reads as "not published".
__global__ void __launch_bounds__(kDB, 2) k_decode(const uint32_t *__restrict__ in, const uint64_t *words_dev,
                                                   uint64_t words_val, uint32_t *__restrict__ out, uint64_t cap,
                                                   uint64_t raw_thr, const uint64_t *n_expect,
                                                   const uint32_t *__restrict__ expect, uint64_t *acc, uint64_t *scal,
                                                   ChunkSlot *slots, uint64_t max_vec, uint64_t max_mb,
                                                   uint64_t *n_out, uint64_t *result, int mode)
{
    extern __shared__ __align__(16) unsigned char s_dyn_d[];
    DecShared &sh = *reinterpret_cast<DecShared *>(s_dyn_d);
    g5_pdl_sync();
    const uint64_t epoch = scal[CS_U_EPOCH];
    const DecHead h = dec_head(in, words_dev ? *words_dev : words_val, cap, raw_thr, n_expect, max_vec, max_mb,
                               gridDim.x);
    uint32_t bad = 0;
    // (as in k_encode)
    const bool lone =
        (!words_dev || words_dev != n_out) && (h.bad || (h.raw ? h.words <= kLoneRaw : h.nchunks <= 1));
    if (lone && blockIdx.x) return;
    if (h.raw) {
        const uint64_t step = lone ? kDB : (uint64_t)gridDim.x * kDB;
        if (!h.bad)
            for (uint64_t i = (uint64_t)blockIdx.x * kDB + threadIdx.x; i < h.words; i += step) {
                const uint32_t x = in[i];
                out[i] = x;
                if (expect && expect[i] != x) bad |= G5_DEVERR_MISMATCH;
            }
    } else if (!h.bad) {
        for (;;) {
            const uint64_t c = lone ? 0 : claim_tile(&scal[CS_U_CTR], &sh.t);
            if (c >= h.nchunks) break;
            bad |= dec_chunk<false>(sh, h, in, c, epoch, slots, &scal[CS_U_ERR], out, cap, expect, mode, &scal[CS_U_N]);
            if (h.nchunks <= gridDim.x) break;  // (as in k_encode)
        }
        if (h.ng == 0 && blockIdx.x == 0 && threadIdx.x < 32) {
            uint64_t n;
            bad |= dec_tail(sh.tail, in, h.words, 4, 0, cap, out, expect, n);
            if (g5_lane() == 0) scal[CS_U_N] = n;
        }
    }
    if (bad) atomicOr((unsigned long long *)&scal[CS_U_ERR], (unsigned long long)bad);
    if (lone) __syncthreads();
    if (lone ? threadIdx.x == 0 : last_block(&scal[CS_U_DONE])) {
        __threadfence();
        uint64_t e = vload64(&scal[CS_U_ERR]), n = vload64(&scal[CS_U_N]);
        if (h.bad) e |= G5_DEVERR_CORRUPT;
        if (h.raw) {
            n = h.words;
            if (n != *n_expect) e |= G5_DEVERR_MISMATCH;
        } else if (e & ~(uint64_t)G5_DEVERR_MISMATCH) {
            n = 0;
        } else if (n_expect && n != *n_expect) {
            e |= G5_DEVERR_MISMATCH;
        }
        scal[CS_ERR] = e;
        scal[CS_N] = n;
        scal[CS_WORDS] = h.words;
        scal[CS_N1] = h.n1;
        if (n_out) *n_out = n;
        if (acc) {
            acc[0] += h.words;
            acc[1] += n;
        }
        if (result) {
            result[0] = n;
            result[1] = h.words;
            result[2] = e;
        }
        scal[CS_U_CTR] = 0;
        scal[CS_U_DONE] = 0;
        scal[CS_U_ERR] = 0;
        scal[CS_U_N] = 0;
        scal[CS_U_EPOCH] = epoch + 1;
        __threadfence();
    }
}

// ---- many streams in one launch -----------------------------------------------------------
//
// The chunks of k queues (or k streams) are numbered one after another and
// claimed in that order; a chunk looks back only at those of its own stream.
// Each stream's bytes are exactly those of a single-stream call.  A raw stream
// is copied kRawChunk values per chunk; a stream without whole miniblocks has
// one chunk, its tail.  Lengths and per-stream errors go straight to pinned
// host memory.
constexpr uint64_t kRawChunk = 8192;

struct EncStream {
    uint64_t in_off, out_off, n;  // first input value, first output word (a multiple of 4), values
    uint32_t t0;                  // its first chunk's number
    uint32_t raw;                 // copied as it is (plugin threshold semantics)
};

struct DecStream {
    uint64_t in_off, out_off, n, words;  // first stream word (a multiple of 4), first output value
    uint32_t t0, nchunks, S;
    uint32_t raw;
};

__device__ __forceinline__ void raw_chunk(const uint32_t *in, uint32_t *out, uint64_t n, uint64_t c)
{
    const uint64_t end = min(n, (c + 1) * kRawChunk);
    for (uint64_t i = c * kRawChunk + threadIdx.x; i < end; i += blockDim.x) out[i] = in[i];
}

__global__ void __launch_bounds__(kEB, 3) k_encode_batch(const uint32_t *__restrict__ in, const EncStream *streams,
                                                      const uint32_t *stream_of, uint32_t chunks, uint32_t gpc,
                                                      uint32_t *__restrict__ out, uint64_t *scal,
                                                      unsigned long long *slots, uint32_t stride, uint64_t *words,
                                                      uint64_t *result, int mode)
{
    extern __shared__ __align__(16) unsigned char s_dyn_e[];
    EncShared &sh = *reinterpret_cast<EncShared *>(s_dyn_e);
    if (threadIdx.x >= 1 && threadIdx.x < 32) sh.magic[threadIdx.x] = 65536u / threadIdx.x + 1u;
    g5_pdl_sync();
    const uint64_t epoch = scal[CS_E_EPOCH];
    for (;;) {
        const uint64_t t = claim_tile(&scal[CS_E_CTR], &sh.t);
        if (t >= chunks) break;
        const uint32_t q = stream_of[t];
        const EncStream st = streams[q];
        const uint64_t c = t - st.t0;
        const uint32_t *x = in + st.in_off;
        uint32_t *o = out + st.out_off;
        if (st.raw) {
            raw_chunk(x, o, st.n, c);
            if (c == 0 && threadIdx.x == 0) words[q] = st.n;
            continue;
        }
        EncLen e = enc_len(st.n, st.n, 0, 1);
        e.gpc = gpc;
        e.nchunks = (e.ng + gpc - 1) / gpc;
        unsigned long long *sl = slots + (uint64_t)stride * st.t0;
        if (e.ng == 0) {
            if (threadIdx.x < 32) {
                const uint64_t w = enc_tail_warp(x, e.n, 0, 4, o, sh.bytes);
                if (threadIdx.x == 0) words[q] = w;
            }
        } else if ((uintptr_t)x & 15) {
            enc_chunk<true>(sh, e, x, c, epoch, sl, stride, &scal[CS_E_ERR], o, mode, words + q);
        } else {
            enc_chunk<false>(sh, e, x, c, epoch, sl, stride, &scal[CS_E_ERR], o, mode, words + q);
        }
    }
    if (last_block(&scal[CS_E_DONE])) {
        __threadfence();
        result[0] = vload64(&scal[CS_E_ERR]);
        scal[CS_E_CTR] = 0;
        scal[CS_E_DONE] = 0;
        scal[CS_E_ERR] = 0;
        scal[CS_E_EPOCH] = epoch + 1;
        __threadfence();
    }
}

// err[q] becomes nonzero for a stream that does not decode to exactly its n
// values (the host cleared it).
__global__ void __launch_bounds__(kDB, 2) k_decode_batch(const uint32_t *__restrict__ in, const DecStream *streams,
                                                      const uint32_t *stream_of, uint32_t chunks,
                                                      uint32_t *__restrict__ out, uint64_t *scal, ChunkSlot *slots,
                                                      uint32_t *err, uint64_t *result, int mode)
{
    extern __shared__ __align__(16) unsigned char s_dyn_d[];
    DecShared &sh = *reinterpret_cast<DecShared *>(s_dyn_d);
    g5_pdl_sync();
    const uint64_t epoch = scal[CS_U_EPOCH];
    for (;;) {
        const uint64_t t = claim_tile(&scal[CS_U_CTR], &sh.t);
        if (t >= chunks) break;
        const uint32_t q = stream_of[t];
        const DecStream st = streams[q];
        const uint64_t c = t - st.t0;
        const uint32_t *x = in + st.in_off;
        uint32_t *o = out + st.out_off;
        if (st.raw) {
            if (st.words == st.n) raw_chunk(x, o, st.n, c);
            else err[q] = 1;
            continue;
        }
        DecHead h;
        h.words = st.words;
        h.nv = st.words / 4;
        h.nmb = st.n / 128;
        h.n1 = h.nmb * 128;
        h.ng = (h.nmb + 15) / 16;
        h.S = st.S;
        h.nchunks = st.nchunks;
        h.raw = false;
        h.bad = st.words < 4;
        if (!h.bad) {
            const uint4 w = *reinterpret_cast<const uint4 *>(x);
            h.bad = w.x != h.n1 || w.y != kCookie || w.z != kCookie || w.w != kCookie;
        }
        // (a stream with groups but no vector for them has no chunk to find it)
        if (h.bad || (h.ng && h.nv < 2)) {
            err[q] = 1;
            continue;
        }
        uint32_t bad = 0;
        uint64_t n = ~0ull;  // the value count, in the lane that decoded the tail
        if (h.ng == 0) {
            if (threadIdx.x < 32) bad = dec_tail(sh.tail, x, h.words, 4, 0, st.n, o, nullptr, n);
        } else if ((uintptr_t)o & 15) {
            bad = dec_chunk<true>(sh, h, x, c, epoch, slots + st.t0, &scal[CS_U_ERR], o, st.n, nullptr, mode, &n);
        } else {
            bad = dec_chunk<false>(sh, h, x, c, epoch, slots + st.t0, &scal[CS_U_ERR], o, st.n, nullptr, mode, &n);
        }
        if (bad || (n != ~0ull && n != st.n)) err[q] = 1;
    }
    if (last_block(&scal[CS_U_DONE])) {
        __threadfence();
        result[0] = vload64(&scal[CS_U_ERR]);
        scal[CS_U_CTR] = 0;
        scal[CS_U_DONE] = 0;
        scal[CS_U_ERR] = 0;
        scal[CS_U_EPOCH] = epoch + 1;
        __threadfence();
    }
}

}  // namespace

size_t codec_bound(size_t n)
{
    const size_t mb = n / 128;
    return 4 + 4 * (mb / 16 + 1) + mb * 128 + ((n % 128) * 5 + 3) / 4 + 8;
}

// chunks of the longest queue, likewise
size_t codec_enc_chunks(size_t max_n)
{
    const size_t groups = (max_n / 128 + 15) / 16;
    return std::min(groups, std::max((size_t)codec_enc_grid(), groups / kEG)) + 2;
}

// chunks of the longest stream: one per block, or as many of the largest size
// as it takes
size_t codec_chunks(size_t max_n)
{
    return std::max((size_t)codec_grid(), (codec_bound(max_n) / 4 + 2) / kMaxChunk) + 2;
}

int codec_grid() { return num_sms() * 2; }
int codec_enc_grid() { return num_sms() * 3; }

g5_status codec_kernels()
{
    G5_CUDA(cudaFuncSetAttribute(k_encode, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(EncShared)));
    G5_CUDA(cudaFuncSetAttribute(k_decode, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DecShared)));
    G5_CUDA(cudaFuncSetAttribute(k_encode_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(EncShared)));
    G5_CUDA(cudaFuncSetAttribute(k_decode_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DecShared)));
    return G5_OK;
}

g5_status codec_work_alloc(CodecWork &w, size_t max_n)
{
    w.max_n = max_n;
    w.max_mb = max_n / 128 + 1;
    w.max_vec = codec_bound(max_n) / 4 + 2;
    w.grid = codec_grid();
    w.egrid = codec_enc_grid();
    const size_t C = codec_chunks(max_n), E = codec_enc_chunks(max_n);
    G5_CUDA(cudaMalloc(&w.scal, sizeof(uint64_t) * kScalars));
    G5_CUDA(cudaMalloc(&w.eslots, 8 * kSlot * E));
    G5_CUDA(cudaMemset(w.eslots, 0, 8 * kSlot * E));
    w.estride = kSlot;
    // more than 48 KB of shared memory each (set per device)
    G5_TRY(codec_kernels());
    G5_CUDA(cudaMalloc(&w.slots, sizeof(ChunkSlot) * C));
    // the decoder's epochs start at 1, so zeroed status words read as "not
    // published" (the encoder's records say so in their low bits)
    G5_CUDA(cudaMemset(w.scal, 0, sizeof(uint64_t) * kScalars));
    G5_CUDA(cudaMemset(w.slots, 0, sizeof(ChunkSlot) * C));
    const uint64_t one = 1;
    G5_CUDA(cudaMemcpy(w.scal + CS_U_EPOCH, &one, sizeof one, cudaMemcpyHostToDevice));
    // a call may be made on a stream that does not wait for the default one
    G5_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    return G5_OK;
}

void codec_work_free(CodecWork &w)
{
    cudaFree(w.scal);
    cudaFree(w.eslots);
    cudaFree(w.slots);
    w = CodecWork();
}

void codec_encode_launch(CodecWork &w, const uint32_t *in, const uint64_t *n_dev, uint64_t n, uint32_t *out, int mode,
                         uint64_t raw_threshold, cudaStream_t s, uint64_t *words_out, uint64_t *result)
{
    // a programmatic dependent launch: the kernel's first instruction waits
    // for the kernel before it, so only the launch latency is overlapped.  A
    // length known here needs no more blocks than it has groups.
    const uint64_t groups = n_dev ? (uint64_t)w.egrid : std::max<uint64_t>(1, (n / 128 + 15) / 16);
    const int grid = (int)std::min<uint64_t>(w.egrid, groups);
    launch_dyn(true, k_encode, grid, kEB, sizeof(EncShared), s, in, n_dev, n, (uint64_t)w.max_n, raw_threshold, out,
               w.scal, w.eslots, w.estride, words_out, result, mode);
}

void codec_decode_launch(CodecWork &w, const uint32_t *in, const uint64_t *words_dev, uint64_t words, uint32_t *out,
                         size_t cap, int mode, uint64_t raw_threshold, const uint64_t *n_expect_dev,
                         const uint32_t *expect, uint64_t *acc, cudaStream_t s, uint64_t *n_out, uint64_t *result)
{
    // a programmatic dependent launch: the kernel's first instruction waits
    // for the kernel before it, so only the launch latency is overlapped.  A
    // length known here needs no more blocks than it has chunks.
    const uint64_t chunks = words_dev ? (uint64_t)w.grid : std::max<uint64_t>(1, (words / 4 + kMinChunk - 1) / kMinChunk);
    const int grid = (int)std::min<uint64_t>(w.grid, chunks);
    launch_dyn(true, k_decode, grid, kDB, sizeof(DecShared), s, in, words_dev, words, out, (uint64_t)cap,
               raw_threshold, n_expect_dev, expect, acc, w.scal, static_cast<ChunkSlot *>(w.slots),
               (uint64_t)w.max_vec, (uint64_t)w.max_mb, n_out, result, mode);
}

}  // namespace g5

// ---- C ABI ----------------------------------------------------------------------------

namespace {

// Buffers of the batched calls, grown on demand (contents not kept).
struct BatchWs {
    void *desc = nullptr, *slots = nullptr;  // device: streams and chunk numbers; records
    void *h_desc = nullptr, *h_res = nullptr;  // pinned: what goes to desc; what the kernel leaves
    size_t desc_cap = 0, slots_cap = 0, res_cap = 0;
    // s: the stream of the launch that will read the records
    g5_status grow(size_t desc_bytes, size_t slot_bytes, size_t res_bytes, cudaStream_t s)
    {
        if (desc_bytes > desc_cap) {
            cudaFree(desc);
            cudaFreeHost(h_desc);
            desc = h_desc = nullptr;
            desc_cap = 0;
            if (cudaMalloc(&desc, desc_bytes) != cudaSuccess || cudaMallocHost(&h_desc, desc_bytes) != cudaSuccess)
                return G5_ERR_OOM;
            desc_cap = desc_bytes;
        }
        if (slot_bytes > slots_cap) {
            cudaFree(slots);
            slots = nullptr;
            slots_cap = 0;
            if (cudaMalloc(&slots, slot_bytes) != cudaSuccess) return G5_ERR_OOM;
            // (zeroed records read as not published; on the launch's own stream,
            // which may not wait for the default one)
            if (cudaMemsetAsync(slots, 0, slot_bytes, s) != cudaSuccess) return G5_ERR_CUDA;
            slots_cap = slot_bytes;
        }
        if (res_bytes > res_cap) {
            cudaFreeHost(h_res);
            h_res = nullptr;
            res_cap = 0;
            if (cudaMallocHost(&h_res, res_bytes) != cudaSuccess) return G5_ERR_OOM;
            res_cap = res_bytes;
        }
        return G5_OK;
    }
    void release()
    {
        cudaFree(desc);
        cudaFree(slots);
        cudaFreeHost(h_desc);
        cudaFreeHost(h_res);
        *this = BatchWs();
    }
};

size_t round4(size_t w) { return (w + 3) & ~(size_t)3; }

}  // namespace

struct g5_codec {
    g5::CodecWork w;
    uint64_t *h_scal = nullptr;  // pinned
    BatchWs be, bd;  // encode, decode
};

extern "C" {

size_t g5_codec_bound(size_t n) { return g5::codec_bound(n); }

g5_status g5_codec_create(size_t max_n, g5_codec **out)
{
    if (!out || max_n == 0 || max_n > ((size_t)1 << 31)) return G5_ERR_INVALID_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return G5_ERR_NO_DEVICE;
    }
    g5_codec *c = new g5_codec();
    g5_status s = g5::codec_work_alloc(c->w, max_n);
    if (s == G5_OK && cudaMallocHost(&c->h_scal, sizeof(uint64_t) * 16) != cudaSuccess) s = G5_ERR_OOM;
    if (s != G5_OK) {
        g5::codec_work_free(c->w);
        delete c;
        return s;
    }
    *out = c;
    return G5_OK;
}

g5_status g5_codec_destroy(g5_codec *c)
{
    if (!c) return G5_ERR_INVALID_ARG;
    cudaDeviceSynchronize();
    g5::codec_work_free(c->w);
    cudaFreeHost(c->h_scal);
    c->be.release();
    c->bd.release();
    delete c;
    return G5_OK;
}

g5_status g5_codec_encode(g5_codec *c, const uint32_t *in_dev, size_t n, uint32_t *out_dev, size_t *out_words,
                          int mode, void *stream)
{
    if (!c || (n && !in_dev) || !out_dev || !out_words || n > c->w.max_n) return G5_ERR_INVALID_ARG;
    if (mode != G5_CODEC_D4 && mode != G5_CODEC_DM) return G5_ERR_INVALID_ARG;
    if (((uintptr_t)in_dev | (uintptr_t)out_dev) & 15) return G5_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    // the kernel leaves the length and status in pinned memory itself
    g5::codec_encode_launch(c->w, in_dev, nullptr, n, out_dev, mode, 0, s, nullptr, c->h_scal);
    G5_CUDA(cudaGetLastError());
    G5_CUDA(cudaStreamSynchronize(s));
    if (c->h_scal[2] & G5_DEVERR_WAIT) return G5_ERR_TIMEOUT;
    if (c->h_scal[2]) return G5_ERR_CAPACITY;
    *out_words = (size_t)c->h_scal[1];
    return G5_OK;
}

g5_status g5_codec_decode(g5_codec *c, const uint32_t *in_dev, size_t words, uint32_t *out_dev, size_t out_cap,
                          size_t *out_n, int mode, void *stream)
{
    if (!c || !in_dev || !out_dev || !out_n) return G5_ERR_INVALID_ARG;
    if (mode != G5_CODEC_D4 && mode != G5_CODEC_DM) return G5_ERR_INVALID_ARG;
    if (((uintptr_t)in_dev | (uintptr_t)out_dev) & 15) return G5_ERR_INVALID_ARG;
    if (words / 4 > c->w.max_vec) return G5_ERR_CAPACITY;
    cudaStream_t s = (cudaStream_t)stream;
    // the kernel leaves the count and status in pinned memory itself
    g5::codec_decode_launch(c->w, in_dev, nullptr, words, out_dev, out_cap, mode, 0, nullptr, nullptr, nullptr, s,
                            nullptr, c->h_scal);
    G5_CUDA(cudaGetLastError());
    G5_CUDA(cudaStreamSynchronize(s));
    if (c->h_scal[2] & G5_DEVERR_WAIT) return G5_ERR_TIMEOUT;
    if (c->h_scal[2]) return G5_ERR_CORRUPT_STREAM;
    *out_n = (size_t)c->h_scal[0];
    return G5_OK;
}

g5_status g5_codec_encode_async(g5_codec *c, const uint32_t *in_dev, const uint64_t *n_dev, uint32_t *out_dev,
                                uint64_t *out_words_dev, int mode, void *stream)
{
    if (!c || !in_dev || !n_dev || !out_dev || !out_words_dev) return G5_ERR_INVALID_ARG;
    if (mode != G5_CODEC_D4 && mode != G5_CODEC_DM) return G5_ERR_INVALID_ARG;
    if (((uintptr_t)in_dev | (uintptr_t)out_dev) & 15) return G5_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    g5::codec_encode_launch(c->w, in_dev, n_dev, 0, out_dev, mode, 0, s, out_words_dev, nullptr);
    G5_CUDA(cudaGetLastError());
    return G5_OK;
}

g5_status g5_codec_decode_async(g5_codec *c, const uint32_t *in_dev, const uint64_t *words_dev, uint32_t *out_dev,
                                size_t out_cap, uint64_t *out_n_dev, int mode, void *stream)
{
    if (!c || !in_dev || !words_dev || !out_dev || !out_n_dev) return G5_ERR_INVALID_ARG;
    if (mode != G5_CODEC_D4 && mode != G5_CODEC_DM) return G5_ERR_INVALID_ARG;
    if (((uintptr_t)in_dev | (uintptr_t)out_dev) & 15) return G5_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    g5::codec_decode_launch(c->w, in_dev, words_dev, 0, out_dev, out_cap, mode, 0, nullptr, nullptr, nullptr, s,
                            out_n_dev, nullptr);
    G5_CUDA(cudaGetLastError());
    return G5_OK;
}

g5_status g5_codec_status(g5_codec *c)
{
    if (!c) return G5_ERR_INVALID_ARG;
    uint64_t err = 0;
    G5_CUDA(cudaMemcpy(&err, c->w.scal + g5::CS_ERR, sizeof err, cudaMemcpyDeviceToHost));
    if (err & G5_DEVERR_WAIT) return G5_ERR_TIMEOUT;
    if (err & G5_DEVERR_CAPACITY) return G5_ERR_CAPACITY;
    if (err) return G5_ERR_CORRUPT_STREAM;
    return G5_OK;
}

size_t g5_codec_batch_bound(const uint64_t *in_off, int k)
{
    if (!in_off || k < 0) return 0;
    size_t w = 0;
    for (int q = 0; q < k; ++q) w += round4(g5::codec_bound((size_t)(in_off[q + 1] - in_off[q])));
    return w;
}

g5_status g5_codec_encode_batch(g5_codec *c, const uint32_t *in_dev, const uint64_t *in_off, int k,
                                uint32_t *out_dev, uint64_t *out_off, uint64_t *out_words,
                                uint32_t raw_threshold, int mode, void *stream)
{
    if (!c || !in_off || !out_off || !out_words || k < 0 || !out_dev) return G5_ERR_INVALID_ARG;
    if (mode != G5_CODEC_D4 && mode != G5_CODEC_DM) return G5_ERR_INVALID_ARG;
    if ((uintptr_t)out_dev & 15) return G5_ERR_INVALID_ARG;
    out_off[0] = 0;
    if (k == 0) return G5_OK;
    if (!in_dev || in_off[0] != 0) return G5_ERR_INVALID_ARG;
    for (int q = 0; q < k; ++q)
        if (in_off[q + 1] < in_off[q]) return G5_ERR_INVALID_ARG;
    if (in_off[k] > ((uint64_t)1 << 31)) return G5_ERR_CAPACITY;  // payload offsets are 32-bit
    // groups per chunk: one chunk per block if that fits, the same for all queues
    uint64_t groups = 0;
    for (int q = 0; q < k; ++q) {
        const uint64_t n = in_off[q + 1] - in_off[q];
        out_off[q + 1] = out_off[q] + round4(g5::codec_bound((size_t)n));
        if (!(raw_threshold && n <= raw_threshold)) groups += (n / 128 + 15) / 16;
    }
    const uint64_t blocks = (uint64_t)c->w.egrid;
    const uint32_t gpc = (uint32_t)std::min<uint64_t>(g5::kEG, std::max<uint64_t>(1, (groups + blocks - 1) / blocks));
    auto chunks_of = [&](uint64_t n, bool raw) -> uint64_t {
        if (raw) return std::max<uint64_t>(1, (n + g5::kRawChunk - 1) / g5::kRawChunk);
        return std::max<uint64_t>(1, ((n / 128 + 15) / 16 + gpc - 1) / gpc);
    };
    uint64_t chunks = 0;
    for (int q = 0; q < k; ++q) {
        const uint64_t n = in_off[q + 1] - in_off[q];
        chunks += chunks_of(n, raw_threshold && n <= raw_threshold);
    }
    if (chunks >= ((uint64_t)1 << 32)) return G5_ERR_CAPACITY;
    BatchWs &w = c->be;
    const size_t sb = sizeof(g5::EncStream) * (size_t)k, db = sb + sizeof(uint32_t) * (size_t)chunks;
    const uint32_t stride = chunks > 16384 ? 2 : g5::kSlot;  // (very many: packed)
    G5_TRY(w.grow(db, sizeof(uint64_t) * stride * (size_t)chunks, sizeof(uint64_t) * ((size_t)k + 1),
                  (cudaStream_t)stream));
    g5::EncStream *hs = static_cast<g5::EncStream *>(w.h_desc);
    uint32_t *ho = reinterpret_cast<uint32_t *>(static_cast<char *>(w.h_desc) + sb);
    uint32_t t = 0;
    for (int q = 0; q < k; ++q) {
        g5::EncStream &b = hs[q];
        b.in_off = in_off[q];
        b.out_off = out_off[q];
        b.n = in_off[q + 1] - in_off[q];
        b.raw = raw_threshold && b.n <= raw_threshold;
        b.t0 = t;
        for (uint64_t e = t + chunks_of(b.n, b.raw != 0); t < e; ++t) ho[t] = (uint32_t)q;
    }
    cudaStream_t s = (cudaStream_t)stream;
    G5_CUDA(cudaMemcpyAsync(w.desc, w.h_desc, db, cudaMemcpyHostToDevice, s));
    uint64_t *hw = static_cast<uint64_t *>(w.h_res);
    const g5::EncStream *ds = static_cast<const g5::EncStream *>(w.desc);
    g5::launch_dyn(true, g5::k_encode_batch, (int)std::min(chunks, blocks), g5::kEB, sizeof(g5::EncShared), s, in_dev, ds,
                   reinterpret_cast<const uint32_t *>(static_cast<const char *>(w.desc) + sb), (uint32_t)chunks, gpc,
                   out_dev, c->w.scal, static_cast<unsigned long long *>(w.slots), stride, hw, hw + k, mode);
    G5_CUDA(cudaGetLastError());
    G5_CUDA(cudaStreamSynchronize(s));
    if (hw[k]) return G5_ERR_TIMEOUT;
    for (int q = 0; q < k; ++q) out_words[q] = hw[q];
    return G5_OK;
}

g5_status g5_codec_decode_batch(g5_codec *c, const uint32_t *in_dev, const uint64_t *in_off,
                                const uint64_t *words, const uint64_t *n, int k, uint32_t *out_dev,
                                uint64_t *out_off, int *stream_ok, uint32_t raw_threshold, int mode,
                                void *stream)
{
    if (!c || !in_off || !words || !n || !out_off || k < 0) return G5_ERR_INVALID_ARG;
    if (mode != G5_CODEC_D4 && mode != G5_CODEC_DM) return G5_ERR_INVALID_ARG;
    out_off[0] = 0;
    if (k == 0) return G5_OK;
    if (!in_dev || !out_dev || ((uintptr_t)in_dev & 15)) return G5_ERR_INVALID_ARG;
    uint64_t total_v = 0;
    for (int q = 0; q < k; ++q) {
        if (in_off[q] % 4) return G5_ERR_INVALID_ARG;  // streams start 16-byte aligned
        // plugin semantics: raw when n <= thr or the stream is as long as n
        const bool raw = raw_threshold && (n[q] <= raw_threshold || words[q] == n[q]);
        out_off[q + 1] = out_off[q] + n[q];
        if (!raw) total_v += words[q] / 4;
    }
    if (total_v >= ((uint64_t)1 << 32) - 2 || out_off[k] > ((uint64_t)1 << 40)) return G5_ERR_CAPACITY;
    const uint64_t blocks = (uint64_t)c->w.grid, per = (total_v + blocks - 1) / blocks;
    auto plan = [&](int q, g5::DecStream &b) -> uint64_t {
        b.in_off = in_off[q];
        b.out_off = out_off[q];
        b.n = n[q];
        b.words = words[q];
        b.raw = raw_threshold && (b.n <= raw_threshold || b.words == b.n);
        const uint64_t nv = b.words / 4, n1 = b.n / 128 * 128;
        b.S = g5::dec_chunk_size(nv, n1, per);
        const uint64_t nc = b.raw ? (b.n + g5::kRawChunk - 1) / g5::kRawChunk : n1 && nv > 1 ? (nv - 1 + b.S - 1) / b.S : 1;
        b.nchunks = (uint32_t)std::max<uint64_t>(1, nc);
        return b.nchunks;
    };
    uint64_t chunks = 0;
    for (int q = 0; q < k; ++q) {
        g5::DecStream b;
        chunks += plan(q, b);
    }
    if (chunks >= ((uint64_t)1 << 32)) return G5_ERR_CAPACITY;
    BatchWs &w = c->bd;
    const size_t sb = sizeof(g5::DecStream) * (size_t)k, db = sb + sizeof(uint32_t) * (size_t)chunks;
    G5_TRY(w.grow(db, sizeof(g5::ChunkSlot) * (size_t)chunks, sizeof(uint64_t) + sizeof(uint32_t) * (size_t)k,
                  (cudaStream_t)stream));
    g5::DecStream *hs = static_cast<g5::DecStream *>(w.h_desc);
    uint32_t *ho = reinterpret_cast<uint32_t *>(static_cast<char *>(w.h_desc) + sb);
    uint32_t t = 0;
    for (int q = 0; q < k; ++q) {
        const uint64_t nc = plan(q, hs[q]);
        hs[q].t0 = t;
        for (uint64_t e = t + nc; t < e; ++t) ho[t] = (uint32_t)q;
    }
    uint64_t *hr = static_cast<uint64_t *>(w.h_res);
    uint32_t *herr = reinterpret_cast<uint32_t *>(hr + 1);
    memset(w.h_res, 0, sizeof(uint64_t) + sizeof(uint32_t) * (size_t)k);
    cudaStream_t s = (cudaStream_t)stream;
    G5_CUDA(cudaMemcpyAsync(w.desc, w.h_desc, db, cudaMemcpyHostToDevice, s));
    const g5::DecStream *ds = static_cast<const g5::DecStream *>(w.desc);
    g5::launch_dyn(true, g5::k_decode_batch, (int)std::min(chunks, blocks), g5::kDB, sizeof(g5::DecShared), s, in_dev, ds,
                   reinterpret_cast<const uint32_t *>(static_cast<const char *>(w.desc) + sb), (uint32_t)chunks, out_dev,
                   c->w.scal, static_cast<g5::ChunkSlot *>(w.slots), herr, hr, mode);
    G5_CUDA(cudaGetLastError());
    G5_CUDA(cudaStreamSynchronize(s));
    bool all = hr[0] == 0;
    for (int q = 0; q < k; ++q) {
        const bool ok = herr[q] == 0;
        if (stream_ok) stream_ok[q] = ok ? 1 : 0;
        all &= ok;
    }
    return all ? G5_OK : (hr[0] & G5_DEVERR_WAIT) ? G5_ERR_TIMEOUT : G5_ERR_CORRUPT_STREAM;
}

}  // extern "C"

// ---- encode without allocation ---------------------------------------------------------
//
// For callers that must not touch the CUDA allocator at all: a serving loop
// that may not block on (or fragment) device memory between requests, or a
// host process whose device memory is owned by another allocator (a
// framework's caching pool) with no headroom for cudaMalloc.  The encoder's
// scratch (its scalars and the record of every chunk) lives in the file-scope
// array below instead of a g5_codec workspace: 8,480 bytes (about 8 KiB,
// kNoAllocBytes) that every GPU which loads the library holds until the
// process exits.  Nothing in it needs clearing between calls: records hold the
// call's epoch.  The array's device address is looked up
// once per device and cached for the life of the process, so the entry point
// must not be used again on a device after cudaDeviceReset in the same
// process (the reset frees the module that holds the array).

namespace {

constexpr size_t kNoAllocMaxValues = (size_t)1 << 20;             // values per call
constexpr size_t kNoAllocChunks = kNoAllocMaxValues / 2048 + 2;   // a chunk is one group at least
constexpr size_t kNoAllocScal = sizeof(uint64_t) * g5::kScalars;  // scalars
constexpr size_t kNoAllocBytes = kNoAllocScal + 16 * kNoAllocChunks;
static_assert(kNoAllocBytes == 8480, "the documented size of the scratch array");

// In host code this name is only a host-side stand-in for the device array;
// kernels receive the device address fetched with cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g5_noalloc_scratch[kNoAllocBytes];

std::mutex g_noalloc_mu;
void *g_noalloc_addr[256] = {nullptr};  // per device ordinal

}  // namespace

extern "C" g5_status g5_codec_encode_noalloc(const uint32_t *in_dev, size_t n, uint32_t *out_dev,
                                             size_t *out_words, int mode, void *stream)
{
    if ((n && !in_dev) || !out_dev || !out_words) return G5_ERR_INVALID_ARG;
    if (mode != G5_CODEC_D4 && mode != G5_CODEC_DM) return G5_ERR_INVALID_ARG;
    if (((uintptr_t)in_dev | (uintptr_t)out_dev) & 15) return G5_ERR_INVALID_ARG;
    if (n > kNoAllocMaxValues) {
        if (getenv("G5_VERBOSE"))
            fprintf(stderr, "g5_codec_encode_noalloc: %zu values exceed the limit of %zu\n", n, kNoAllocMaxValues);
        return G5_ERR_CAPACITY;
    }
    int dev = 0;
    G5_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 256) return G5_ERR_INVALID_ARG;
    void *base = nullptr;
    {
        // set-up, once per device, with that device current
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_addr[dev]) {
            void *p = nullptr;
            G5_CUDA(cudaGetSymbolAddress(&p, g5_noalloc_scratch));
            G5_TRY(g5::codec_kernels());
            g_noalloc_addr[dev] = p;
        }
        base = g_noalloc_addr[dev];
    }
    unsigned char *b = static_cast<unsigned char *>(base);
    g5::CodecWork w;
    w.max_n = kNoAllocMaxValues;
    w.egrid = g5::codec_enc_grid();
    w.scal = reinterpret_cast<uint64_t *>(b);
    w.eslots = reinterpret_cast<unsigned long long *>(b + kNoAllocScal);
    w.estride = 2;  // packed: the array is kept small
    static_assert(kNoAllocScal % 16 == 0, "records are 16-byte vectors");
    cudaStream_t s = (cudaStream_t)stream;
    g5::codec_encode_launch(w, in_dev, nullptr, n, out_dev, mode, 0, s, nullptr, nullptr);
    G5_CUDA(cudaGetLastError());
    uint64_t sc[3] = {0, 0, 0};  // CS_N, CS_WORDS, CS_ERR
    G5_CUDA(cudaMemcpyAsync(sc, w.scal, sizeof sc, cudaMemcpyDeviceToHost, s));
    G5_CUDA(cudaStreamSynchronize(s));
    if (sc[g5::CS_ERR] & G5_DEVERR_WAIT) return G5_ERR_TIMEOUT;
    if (sc[g5::CS_ERR]) return G5_ERR_CAPACITY;
    *out_words = (size_t)sc[g5::CS_WORDS];
    return G5_OK;
}
