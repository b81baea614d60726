// The Fiat-Shamir transcript on the device, for stretches of the protocol that run without the
// host: the sumcheck round loops, whose every round is a kernel's sums -> round polynomial ->
// proof message -> challenge -> the next kernel's fold.  Run on the host, each round costs a
// device-to-host round trip; run here, a loop is a chain of launches the host enqueues at once.
//
// The state is the host Transcript's own (TranscriptState): the same HasherChallenger rules
// (verifier/transcript/src/fiat_shamir/hasher_challenger.rs:14-200) over the same SHA-256 stream,
// so a stretch may start and end anywhere in the protocol and the proof bytes do not change.  A
// device stretch is advanced by one warp whose lanes hold the same state (the steps are a strict
// chain; the lanes share the multiplies, see gf_mul_warp); message bytes go to a device tape that
// the host appends to the proof when the stretch ends.
#pragma once
#include <stdint.h>

#include <initializer_list>
#include <vector>

#include "gf128.cuh"
#include "internal.h"
#include "sha256.cuh"
#include "transcript.h"

namespace bgpu {

// The scalar protocol steps run on one warp, where every dependent instruction waits out its full
// latency and every logic instruction takes the warp's 16-lane pipe for two cycles.  Measured on a
// B200, one warp: the multiply below 0.13 us (a 32x32 carry-less product per lane and eight warp
// reductions: 0.37 us; one thread: 0.67 us); a SHA-256 compression fully unrolled on registers 1.5
// us.  The steps of a stretch run as FsStep below (2.4 us for message and challenge).

// A product on the critical path of a Fiat-Shamir step, computed by a whole warp.  One out-of-line
// copy keeps the code of the launches that call it small.
static __device__ __noinline__ uint4 gf_mul_warp(uint4 a, uint4 b) { return gf_mul_lanes(a, b); }

// One compression of blk into st, both held in local memory by the caller: copied to registers,
// compressed by the fully unrolled sha256_compress (round constants as immediates) and written
// back.  One out-of-line copy serves every call site.
static __device__ __noinline__ void sha256_compress_1t(uint32_t* st, const uint32_t* blk) {
  uint32_t s[8], w[16];
#pragma unroll
  for (int i = 0; i < 8; i++) s[i] = st[i];
#pragma unroll
  for (int i = 0; i < 16; i++) w[i] = blk[i];
  sha256_compress(s, w);
#pragma unroll
  for (int i = 0; i < 8; i++) st[i] = s[i];
}

// The challenger held by a thread that adds a message without a challenge after it.  The partial
// SHA-256 block is kept as 16 big-endian words, the sample buffer as 8 little-endian words;
// absorbing a word is one store at a run-time index (the arrays live in local memory, which the
// out-of-line compression copies to registers), so the code around the compression stays small.  The
// stream is absorbed in 4-byte pieces (every message of the protocol is a whole number of words); a piece
// may start at any byte offset.  Words at or past `len` hold no meaning except that a partially
// filled word is zero past its bytes.
struct DevTr {
  uint32_t h[8], w[16], len;  // chaining value, partial block, bytes in it
  uint64_t total;             // bytes absorbed since the last reset
  uint32_t sampling, index;   // mode and bytes of buf consumed
  uint32_t buf[8];            // sample buffer, little-endian words
  uint32_t tape_len, tape_cap, error;

  static __device__ __forceinline__ void compress(uint32_t* st, const uint32_t* blk) {
    sha256_compress_1t(st, blk);
  }

  __device__ __forceinline__ void load(const TranscriptState* g) {
    for (int i = 0; i < 8; i++) h[i] = g->h[i];
    for (int i = 0; i < 16; i++) w[i] = g->w[i];
    len = g->block_len & 63u;
    total = g->total;
    sampling = g->sampling;
    index = g->index;
    for (int i = 0; i < 8; i++) buf[i] = g->buf[i];
    tape_len = g->tape_len;
    tape_cap = g->tape_cap;
    error = g->error;
  }

  __device__ __forceinline__ void store(TranscriptState* g) const {
    for (int i = 0; i < 8; i++) g->h[i] = h[i];
    for (int i = 0; i < 16; i++) g->w[i] = w[i];
    g->block_len = len;
    g->total = total;
    g->sampling = sampling;
    g->index = index;
    for (int i = 0; i < 8; i++) g->buf[i] = buf[i];
    g->tape_len = tape_len;
    g->tape_cap = tape_cap;
    g->error = error;
  }

  // Absorbs 4 stream bytes given as a little-endian word (first byte lowest).
  __device__ __noinline__ void absorb_word(uint32_t le) {
    const uint32_t be = bswap32(le);
    const uint32_t off = len & 3u;
    total += 4;
    if (off == 0) {
      w[len >> 2] = be;
      len += 4;
      if (len == 64) {
        compress(h, w);
        len = 0;
      }
    } else {
      w[len >> 2] |= be >> (8 * off);
      len += 4 - off;
      if (len == 64) {
        compress(h, w);
        len = 0;
      }
      w[len >> 2] = be << (8 * (4 - off));
      len += off;
    }
  }

  __device__ __forceinline__ void to_observer() {
    if (sampling) {
      const uint32_t idx = index;
      absorb_word(idx);
      absorb_word(0u);
      sampling = 0;
    }
  }

  // Appends n whole words (little-endian) to the tape; sets error instead when they do not fit.
  __device__ __forceinline__ void tape_words(uint8_t* tape, const uint32_t* v, uint32_t n) {
    if (tape_len + 4 * n > tape_cap) {
      error = 1;
      return;
    }
    if ((tape_len & 3u) == 0) {
      uint32_t* t32 = reinterpret_cast<uint32_t*>(tape + tape_len);
      for (uint32_t i = 0; i < n; i++) t32[i] = v[i];
    } else {
      for (uint32_t i = 0; i < 4 * n; i++)
        tape[tape_len + i] = (uint8_t)(v[i >> 2] >> (8 * (i & 3)));
    }
    tape_len += 4 * n;
  }

  // message(): n words to the tape and the challenger.
  __device__ __forceinline__ void message_words(uint8_t* tape, const uint32_t* v, uint32_t n) {
    tape_words(tape, v, n);
    if (n) {
      to_observer();
      if ((len & 3u) == 0) {  // word-aligned stream (every message of the protocol): inline
        for (uint32_t i = 0; i < n; i++) {
          w[len >> 2] = bswap32(v[i]);
          len += 4;
          if (len == 64) {
            compress(h, w);
            len = 0;
          }
        }
        total += 4ull * n;
      } else {
        for (uint32_t i = 0; i < n; i++) absorb_word(v[i]);
      }
    }
  }
};

// A round's Fiat-Shamir step, message() of n elements then sample(), by three warps of a block.
//
// Between the rounds of a stretch the transcript is in one state: it has just been sampled, so the
// SHA-256 stream holds the 32 bytes of the last digest and nothing else.  From there a step absorbs those, 8 bytes for the return to observing and the message, and digests
// the padded stream: two blocks, whose words are all known before the first compression.  Warp 0
// lays the words out (one per lane) and runs the 64 + 64 rounds; warps 1 and 2, on other
// schedulers, expand the two message schedules meanwhile and hand them over through shared memory
// with the round constants added.  A compression on one warp is bound by that warp's logic pipe
// (1376 instructions of two cycles); without the schedules 900 are left.  Measured, one step:
// 2.4 us against 4.9 us on one warp; a 2^12-word proof 2.55 -> 2.20 ms, one of 2^18 words and 256
// multiplications 5.30 -> 4.46 ms, one of 2^20 words 3.04 -> 2.78 ms (with the multiply above).
// A stretch begins in that state: DeviceTranscript::check has the host sample first.
constexpr uint32_t kFsThreads = 96;  // warps 0, 1 and 2 take part
struct __align__(16) FsShared {
  uint32_t words[32];   // the stream's two padded blocks; between steps the digest in 0..7
  uint32_t kw[2][64];   // their schedules plus round constants
};

// Named barriers of a step; 0 is __syncthreads.
constexpr uint32_t kFsWords = 8, kFsSecond = 12;  // 9, 10, 11: 16 schedule words each
__device__ __forceinline__ void fs_wait(uint32_t id, uint32_t threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void fs_arrive(uint32_t id, uint32_t threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// 64 rounds on s from schedule words with their constants added, 16 at a time; with `chunked`
// the words past the first 16 are waited for as they come.
__device__ __forceinline__ void fs_rounds(uint32_t (&s)[8], const uint32_t* kw, bool chunked) {
  uint32_t a = s[0], b = s[1], c = s[2], d = s[3], e = s[4], f = s[5], g = s[6], h = s[7];
#pragma unroll 1
  for (uint32_t it = 0; it < 4; it++) {
    if (chunked && it) fs_wait(kFsWords + it, 64);
    uint4 k4[4];
#pragma unroll
    for (int i = 0; i < 4; i++) k4[i] = reinterpret_cast<const uint4*>(kw + 16 * it)[i];
    const uint32_t* k = reinterpret_cast<const uint32_t*>(k4);
#pragma unroll
    for (int t = 0; t < 16; t++) {
      const uint32_t S1 = rotr32(e, 6) ^ rotr32(e, 11) ^ rotr32(e, 25);
      const uint32_t ch = (e & f) ^ (~e & g);
      const uint32_t S0 = rotr32(a, 2) ^ rotr32(a, 13) ^ rotr32(a, 22);
      const uint32_t mj = (a & b) ^ (a & c) ^ (b & c);
      const uint32_t y = ch + (h + k[t]);
      const uint32_t ne = (d + y) + S1, na = (y + S1) + (S0 + mj);
      h = g;
      g = f;
      f = e;
      e = ne;
      d = c;
      c = b;
      b = a;
      a = na;
    }
  }
  s[0] += a;
  s[1] += b;
  s[2] += c;
  s[3] += d;
  s[4] += e;
  s[5] += f;
  s[6] += g;
  s[7] += h;
}

// Warp 1 (block = 0) and warp 2 (block = 1) of a step.
static __device__ __noinline__ void fs_schedule(FsShared& sh, uint32_t block) {
  fs_wait(kFsWords, kFsThreads);
  uint32_t w[16];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint4 v = reinterpret_cast<const uint4*>(sh.words + 16 * block)[i];
    w[4 * i] = v.x;
    w[4 * i + 1] = v.y;
    w[4 * i + 2] = v.z;
    w[4 * i + 3] = v.w;
  }
#pragma unroll 1
  for (uint32_t it = 1; it < 4; it++) {
    uint32_t o[16];
#pragma unroll
    for (int t = 0; t < 16; t++) {
      const uint32_t w15 = w[(t + 1) & 15], w2 = w[(t + 14) & 15];
      const uint32_t s0 = rotr32(w15, 7) ^ rotr32(w15, 18) ^ (w15 >> 3);
      const uint32_t s1 = rotr32(w2, 17) ^ rotr32(w2, 19) ^ (w2 >> 10);
      w[t] = w[t] + s0 + w[(t + 9) & 15] + s1;
      o[t] = w[t] + kSha256K[16 * it + t];
    }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
      for (int i = 0; i < 4; i++)
        reinterpret_cast<uint4*>(sh.kw[block] + 16 * it)[i] =
            make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
    }
    if (block == 0) fs_arrive(kFsWords + it, 64);
  }
  if (block) fs_arrive(kFsSecond, 64);
}

// Warp 0's side: every lane holds the same values.
struct FsStep {
  uint32_t k16;  // round constant lane mod 16
  uint32_t index, tape_len, tape_cap, error;

  __device__ __forceinline__ void begin(FsShared& sh, const TranscriptState* g) {
    const uint32_t lane = threadIdx.x & 31;
    k16 = kSha256K[lane & 15];
    index = g->index;
    tape_len = g->tape_len;
    tape_cap = g->tape_cap;
    error = g->error;
    if (lane < 8) sh.words[lane] = g->w[lane];
  }

  // n <= 4 elements.
  __device__ __forceinline__ uint4 step(FsShared& sh, uint8_t* tape, const uint4* msg, uint32_t n) {
    const uint32_t lane = threadIdx.x & 31;
    if (lane == 0) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        if ((uint32_t)e >= n) break;
        uint2* w = reinterpret_cast<uint2*>(sh.words + 10 + 4 * e);
        w[0] = make_uint2(bswap32(msg[e].x), bswap32(msg[e].y));
        w[1] = make_uint2(bswap32(msg[e].z), bswap32(msg[e].w));
      }
    }
    __syncwarp();
    const uint32_t end = 10 + 4 * n;
    uint32_t x = sh.words[lane];
    if (lane == 8) x = bswap32(index);
    if (lane == 9) x = 0;
    if (tape_len + 16 * n > tape_cap) {
      error = 1;
    } else {
      if (lane >= 10 && lane < end) {
        const uint32_t at = tape_len + 4 * (lane - 10);
        if ((tape_len & 3u) == 0) {
          *reinterpret_cast<uint32_t*>(tape + at) = bswap32(x);
        } else {
          for (int i = 0; i < 4; i++) tape[at + i] = (uint8_t)(x >> (24 - 8 * i));
        }
      }
      tape_len += 16 * n;
    }
    if (lane == end) x = 0x80000000u;
    if (lane > end) x = lane == 31 ? 32 * end : 0u;
    sh.words[lane] = x;
    sh.kw[lane >> 4][lane & 15] = x + k16;
    fs_wait(kFsWords, kFsThreads);
    uint32_t s[8];
    sha256_init(s);
    fs_rounds(s, sh.kw[0], true);
    fs_wait(kFsSecond, 64);
    fs_rounds(s, sh.kw[1], false);
    if (lane == 0) {
      reinterpret_cast<uint4*>(sh.words)[0] = make_uint4(s[0], s[1], s[2], s[3]);
      reinterpret_cast<uint4*>(sh.words)[1] = make_uint4(s[4], s[5], s[6], s[7]);
    }
    __syncwarp();
    index = 16;
    return make_uint4(bswap32(s[0]), bswap32(s[1]), bswap32(s[2]), bswap32(s[3]));
  }

  // After at least one step.  Writes every field but tape_cap.
  __device__ __forceinline__ void end(const FsShared& sh, TranscriptState* g) const {
    const uint32_t lane = threadIdx.x & 31;
    if (lane < 8) {
      uint32_t iv[8];
      sha256_init(iv);
      uint32_t v = iv[0];
#pragma unroll
      for (int i = 1; i < 8; i++) v = lane == (uint32_t)i ? iv[i] : v;
      g->h[lane] = v;
      g->buf[lane] = bswap32(sh.words[lane]);
    }
    if (lane < 16) g->w[lane] = lane < 8 ? sh.words[lane] : 0u;
    if (lane == 0) {
      g->block_len = 32;
      g->total = 32;
      g->sampling = 1;
      g->index = index;
      g->tape_len = tape_len;
      g->error = error;
    }
  }
};

// The other warps of the block during a step.
__device__ __forceinline__ void fs_help(FsShared& sh) {
  const uint32_t warp = threadIdx.x / 32;
  if (warp == 1 || warp == 2) fs_schedule(sh, warp - 1);
}

// The products of a small sumcheck round in one block: job(j, mul, own) for j < n, on threads
// (mul a thread's product; own = true) or, when no more than the block's warps, each on a warp of
// its own whose lanes all run it (mul a warp's product, a fifth of the latency; own on lane 0).
// Warp 0, which also runs the Fiat-Shamir step and its algebra, comes last.
template <class Job>
__device__ __forceinline__ void block_jobs(uint32_t n, const Job& job) {
  const uint32_t warps = blockDim.x >> 5;
  if (n <= warps) {
    const uint32_t j = warps - 1 - (threadIdx.x >> 5);
    if (j < n)
      job(j, [](uint4 a, uint4 b) { return gf_mul_warp(a, b); }, (threadIdx.x & 31) == 0);
  } else {
    const uint32_t first = threadIdx.x >= 32 ? threadIdx.x - 32 : threadIdx.x + blockDim.x - 32;
    for (uint32_t j = first; j < n; j += blockDim.x)
      job(j, [](uint4 a, uint4 b) { return gf_mul_nl(a, b); }, true);
  }
}

// Host side of one device stretch.  begin() hands the host transcript's state to the device;
// kernels advance state() and write to tape(); read() queues the copy-back of the state and of
// the `tape_bytes` the stretch is known to write, and finish() (after the reads were waited on)
// hands the state back to the host transcript with those bytes appended.
class DeviceTranscript {
 public:
  static constexpr uint32_t kTapeCap = 1u << 16;

  ~DeviceTranscript();
  // With the state, `uploads` from host memory to 16-byte aligned device memory.
  struct Upload {
    void* dst;
    const void* src;
    size_t bytes;
  };
  int begin(const Transcript& t, cudaStream_t s, std::initializer_list<Upload> uploads = {});
  // A state that FsStep can go on from: just sampled (the stream is the last digest, 32 bytes).
  static int check(const TranscriptState& st);
  TranscriptState* state() const { return reinterpret_cast<TranscriptState*>(mem_); }
  uint8_t* tape() const { return mem_ + kStateBytes; }
  // message() of n_bytes (a multiple of 4, 4-byte aligned) that are in device memory.
  int message_device(const void* d_bytes, uint32_t n_bytes, cudaStream_t s);
  int read(StagedReads& rd, uint32_t tape_bytes);
  int finish(Transcript& t);

 private:
  static constexpr size_t kStateBytes = 256;
  cudaStream_t s_ = nullptr;
  uint8_t* mem_ = nullptr;
  uint32_t expect_ = 0;
  TranscriptState host_state_;
  std::vector<uint8_t> host_tape_;
};

}  // namespace bgpu
