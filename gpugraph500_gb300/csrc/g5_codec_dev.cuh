// g5_codec_dev.cuh -- device-resident s4-bp128 codec pipeline, callable from
// a BFS level loop (lengths live in device memory, grids are fixed, so the
// launches can be captured in a CUDA graph).
#pragma once

#include <cstdint>

#include "g5_common.cuh"

namespace g5 {

// Four running lane sums and a reset flag (a raw miniblock restarts the sums).
struct VecFlag {
    uint4 v;
    uint32_t f;
};

struct CodecWork {
    size_t max_n = 0;        // capacity in values
    size_t max_mb = 0;       // miniblocks
    size_t max_vec = 0;      // 16-byte vectors of the largest stream
    int grid = 0, egrid = 0; // blocks of the decoder's and encoder's fixed grids
    uint64_t *scal = nullptr;  // device scalars (kScalars), see CodecScalar
    unsigned long long *eslots = nullptr;  // encoder: a record (16 bytes) per chunk,
    uint32_t estride = 0;                  // this many 64-bit words apart
    void *slots = nullptr;     // decoder: a record per chunk
};

enum CodecScalar {
    CS_N = 0,       // values to encode / decoded value count
    CS_WORDS = 1,   // encoded words
    CS_ERR = 2,     // error bits (G5_DEVERR_*)
    CS_N1 = 3,      // values in the block part
    CS_COUNT = 8
};

constexpr int kScalars = 32;  // scalar slots of a CodecWork

// The fixed grids of the decoder and the encoder, and their attributes on the
// current device.
int codec_grid();
int codec_enc_grid();
g5_status codec_kernels();

size_t codec_bound(size_t n);
g5_status codec_work_alloc(CodecWork &w, size_t max_n);
void codec_work_free(CodecWork &w);

// Encode in[0 .. *n_dev) (or [0 .. n) if n_dev is null) to out; words written
// -> w.scal[CS_WORDS] and, if given, *words_out; result (pinned host memory, 3
// entries) receives the length, the words and the error bits.  raw_threshold:
// if the length is at most that, a raw copy (plugin semantics); pass 0 for pure
// IntegerCODEC semantics.
void codec_encode_launch(CodecWork &w, const uint32_t *in, const uint64_t *n_dev, uint64_t n, uint32_t *out, int mode,
                         uint64_t raw_threshold, cudaStream_t s, uint64_t *words_out, uint64_t *result);

// Decode in[0 .. *words_dev) (or [0 .. words) if words_dev is null) to out
// (capacity cap); values -> w.scal[CS_N].  If expect != nullptr, each decoded
// value is compared with expect[i] and *n_expect_dev with the decoded count; a
// difference sets G5_DEVERR_MISMATCH.  raw_threshold as for encode (raw when
// n <= thr or words == n), with *n_expect_dev giving the original length.  If
// given, acc[0] += words and acc[1] += decoded values (running totals kept on
// the device), n_out receives the value count, and result (pinned host
// memory, 3 entries) the count, the words and the error bits.
void codec_decode_launch(CodecWork &w, const uint32_t *in, const uint64_t *words_dev, uint64_t words, uint32_t *out,
                         size_t cap, int mode, uint64_t raw_threshold, const uint64_t *n_expect_dev,
                         const uint32_t *expect, uint64_t *acc, cudaStream_t s, uint64_t *n_out, uint64_t *result);

}  // namespace g5
