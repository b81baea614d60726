// GF(2^128) multiplication of many elements by ONE element on the tcgen05 tensor cores.
//
// x -> t x is a linear map of the 128 bits of x over GF(2): bit n of t x is the parity of
// sum_j M[n][j] x_j with M[n][j] = bit n of t x^j.  A tile of 128 elements is therefore one
// 128 x 128 x 128 matrix product whose entries are zero or one and whose sums are at most 128,
// followed by taking the parity of every sum.  It runs as two kind::mxf4 instructions
// (M = 128 elements, N = 128 output bits, K = 64 input bits each), exact in f32:
//
// * A (the elements) lies in tensor memory, one element per lane, so a thread writes its own
//   element's operand row and reads its own sums.  The operand nibbles are masks of the element's
//   words: w & (0x11111111 << k) leaves bit k of each nibble in place, and a lone bit in position
//   k < 3 is an e2m1 power of two, 0.5, 1, 2 for k = 0, 1, 2 (bit 3, the sign, is moved to
//   position 2).  One or two logic instructions make eight operand nibbles.
// * B (the matrix of t) lies in shared memory, its entries the reciprocals: 2, 1, 0.5, 0.5.  Its
//   block scales, kept in tensor memory, multiply row n by 2^(-12 + n mod 8).
// * The sums of rows n and n + 8 (n mod 16 < 8) share one f32: the second comes with a scale 2^8
//   larger, onto the same accumulator, and a first product of ones adds 2^11, whose ulp is 2^-12.
//   So the sum's mantissa holds count_n at bits j..j+7 and count_(n+8) at bits j+8..j+15,
//   j = n mod 8, exactly: 24 bits in all.  The two parities sit at bits j and j + 8 of the word,
//   and sixteen output bits are gathered from eight words by seven bit selects.
//
// An element times a SUM of multipliers chosen by bits of its row (t_0 + sum of bit_j t_j) takes
// one more operand slot and matrix per bit: the slot holds the element where the bit is set and
// zero elsewhere, and the products accumulate.  Counts then pass 255, so a sum has one row only,
// and the output bits are formed in two halves.
//
// Measured on B200 at 1965 MHz: 161 cycles of the tensor pipe per 128 products, exact over random
// and all-ones elements (with e4m3 / e5m2 operands 258, and matrices of twice the size).  The
// ~100 logic instructions per product that write the operand and gather the sums bound it.
#pragma once
#include "gf128.cuh"

namespace bgpu {
namespace tc {

constexpr uint32_t kGroupThreads = 128;         // a group works on tiles of 128 elements
constexpr uint32_t kMatrixBytes = 128 * 64;     // the operand matrix of one multiplier
constexpr uint32_t kSumCols = 64;               // TMEM columns of a tile's sums
constexpr uint32_t kOperandCols = 16;           // TMEM columns of a tile's operand
constexpr uint32_t kConstCols = 24;             // TMEM columns of the scales and the ones
constexpr uint32_t kOnesBytes = 64 * 64;        // shared memory of the ones

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// x of lane 0 of the (converged) warp: makes a value the compiler cannot see as uniform uniform,
// so that the tensor instructions take it from uniform registers (a tile's four instructions and
// their commit issue in 45 cycles so, in 220 from a divergent thread).
__device__ __forceinline__ uint32_t uniform(uint32_t x) { return __shfl_sync(0xffffffffu, x, 0); }

// ---- tensor memory (one warp; it frees what it allocated)
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_addr(smem_dst)),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Shared-memory writes of this thread before it, tensor-core reads of them after a barrier.
__device__ __forceinline__ void fence_smem_to_tensor() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Named barrier of a group: its writes are seen by the warps that wait; the others go on.  A warp
// may arrive again only when the barrier has completed (say, because what it guarded has).
__device__ __forceinline__ void group_arrive(uint32_t id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kGroupThreads) : "memory");
}
__device__ __forceinline__ void group_wait(uint32_t id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kGroupThreads) : "memory");
}

// ---- completion barriers
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t arrivals) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(arrivals)
               : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done;
}
// Waits for the phase of this parity: a bounded number of polls, each of which may sleep for some
// 20 us, far beyond any tile's time.  `ok` becomes false when they run out; the thread then polls
// once or twice a wait, goes through the rest of its launch (what it stores means nothing) and
// reports at the end (finish_launch).
constexpr uint32_t kWaitPolls = 1u << 16;
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, bool& ok,
                                          uint32_t polls = kWaitPolls) {
  const uint32_t a = smem_addr(bar);
  if (mbar_try(a, parity)) return;
  for (uint32_t left = ok ? polls : 1; left; left--)
    if (mbar_try(a, parity)) return;
  ok = false;
}
// Reports a wait that ran out (tensor_word in internal.h).
__device__ __forceinline__ void report_stall(uint32_t* word) {
  *static_cast<volatile uint32_t*>(word) = 1;
  __threadfence_system();
}

// ---- the multiplier's matrix
//
// Row n holds, at bit j, bit n of t x^j mod x^128 + x^7 + x^2 + x + 1.  Coefficient i of the
// unreduced t x^j is t_(i-j); coefficient 128 + m folds into m, m + 1, m + 2 and m + 7, and the
// few of those at or past 128 once more.  With rt the reversed bits of t and
// Q = rt + rt<<5 + rt<<6 + rt<<7, every row is the window of 128 bits at 127 - n of the 256-bit
// string rt + Q<<121, but for the rows below 13: below 7 the string holds folds that would come
// from below coefficient 128, and the second folds (of coefficients 128..133) are missing.

struct MatrixRows {
  uint4 window[2];  // the string
  uint4 low[13];    // rows 0..12
};
// What matrix_build reads of t: 14 items, which any threads may write, then a barrier.
constexpr uint32_t kRowItems = 14;
__device__ __forceinline__ void matrix_rows(MatrixRows& dst, uint4 t, uint32_t item) {
  const uint32_t r[4] = {__brev(t.w), __brev(t.z), __brev(t.y), __brev(t.x)};
  uint32_t q[4];
  q[0] = r[0] ^ (r[0] << 5) ^ (r[0] << 6) ^ (r[0] << 7);
#pragma unroll
  for (int i = 1; i < 4; i++)
    q[i] = r[i] ^ __funnelshift_l(r[i - 1], r[i], 5) ^ __funnelshift_l(r[i - 1], r[i], 6) ^
           __funnelshift_l(r[i - 1], r[i], 7);
  const uint32_t s[8] = {r[0],
                         r[1],
                         r[2],
                         r[3] ^ (q[0] << 25),
                         __funnelshift_l(q[0], q[1], 25),
                         __funnelshift_l(q[1], q[2], 25),
                         __funnelshift_l(q[2], q[3], 25),
                         __funnelshift_l(q[3], (r[3] >> 27) ^ (r[3] >> 26) ^ (r[3] >> 25), 25)};
  if (item == 13) {
    dst.window[0] = make_uint4(s[0], s[1], s[2], s[3]);
    dst.window[1] = make_uint4(s[4], s[5], s[6], s[7]);
    return;
  }
  const uint32_t n = item, sh = 31 - n;  // 127 - n = 96 + sh
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; i++) w[i] = __funnelshift_r(s[3 + i], s[4 + i], sh);
  const uint32_t taps[4] = {0, 1, 2, 7};
#pragma unroll
  for (int d = 0; d < 4; d++) {
    if (taps[d] > n) {  // take the fold from coefficient 128 + n - tap < 128 out
      const uint32_t u = taps[d] - n - 1;
      w[0] ^= __funnelshift_r(r[0], r[1], u);
      w[1] ^= __funnelshift_r(r[1], r[2], u);
      w[2] ^= __funnelshift_r(r[2], r[3], u);
      w[3] ^= r[3] >> u;
    } else if (n - taps[d] <= 5) {  // the second fold of coefficient 128 + u
      const uint32_t u = n - taps[d];
      w[3] ^= r[0] << (26 + u);
      if (u == 0) w[3] ^= r[0] << 31;
    }
  }
  dst.low[n] = make_uint4(w[0], w[1], w[2], w[3]);
}

// Writes row n (of 128) of a matrix; the 128 threads of a group build a matrix together, then
// fence_smem_to_tensor() and a barrier.  Layout: first the rows with n mod 16 < 8, then the
// others, each part K-major without swizzle in 8-row x 16-byte core matrices, the four of a row
// block consecutive.  K position 32 q + 8 k + b is input bit 32 q + 4 b + k, the order in which
// operand_words lays an element's bits out.
__device__ __forceinline__ void matrix_build(uint8_t* m, const MatrixRows& rows, uint32_t n) {
  uint32_t w[4];
  {
    const uint32_t* ws = reinterpret_cast<const uint32_t*>(rows.window) + ((127 - n) >> 5);
    const uint32_t sh = (127 - n) & 31;
    uint32_t lo = ws[0];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t hi = ws[i + 1];
      w[i] = __funnelshift_r(lo, hi, sh);
      lo = hi;
    }
  }
  if (n < 13) {
    const uint4 x = rows.low[n];
    w[0] = x.x;
    w[1] = x.y;
    w[2] = x.z;
    w[3] = x.w;
  }
  uint4* dst = reinterpret_cast<uint4*>(m + ((n >> 3) & 1) * (kMatrixBytes / 2) + (n >> 4) * 512 +
                                        (n & 7) * 16);
#pragma unroll
  for (int q = 0; q < 4; q++)
    dst[8 * q] = make_uint4((w[q] << 2) & 0x44444444u, w[q] & 0x22222222u,
                            (w[q] >> 2) & 0x11111111u, (w[q] >> 3) & 0x11111111u);
}

// Writes the constants: in tensor memory (kConstCols columns at tmem, this warp's lanes) ones for
// the elements' scales at column 0, 2^(-12 + n mod 8) for the first rows at 4, 2^8 times that at 6,
// 2^11 for the ones at 8 (row r's scale sits in lane r mod 32 of column r / 32, one e8m0 byte per
// block of 32 along K), and the operand of the ones at 12; in shared memory (kOnesBytes) their
// matrix.  The 128 threads of a group call it; then fence_smem_to_tensor() and a barrier.
__device__ __forceinline__ void constants_store(uint32_t tmem, uint8_t* ones) {
  const uint32_t one = 0x7f7f7f7fu;
  const uint32_t first = (127 - 12 + (threadIdx.x & 7)) * 0x01010101u;
  const uint32_t second = first + 8 * 0x01010101u;
  const uint32_t bias = (127 + 11) * 0x01010101u;
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%2,%2,%3,%3,%4,%4,%4,%4,%5,%6,%6,"
      "%6};\n"
      "tcgen05.st.sync.aligned.32x32b.x4.b32 [%7], {%6,%6,%6,%6};" ::"r"(tmem),
      "r"(one), "r"(first), "r"(second), "r"(bias), "r"(2u), "r"(0u), "r"(tmem + 16)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  const uint32_t t = threadIdx.x % kGroupThreads;
  for (uint32_t i = t; i < kOnesBytes / 16; i += kGroupThreads) {
    const bool k0 = (i & 31) < 8;  // K block 0 of its row block: nibble 0 is 1
    reinterpret_cast<uint4*>(ones)[i] = make_uint4(k0 ? 2u : 0u, 0u, 0u, 0u);
  }
}

// ---- one tile: operand in, products, sums out
// The operand row of element x.
__device__ __forceinline__ void operand_words(uint4 x, uint32_t (&r)[16]) {
  const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int q = 0; q < 4; q++) {
#pragma unroll
    for (int k = 0; k < 3; k++) r[4 * q + k] = w[q] & (0x11111111u << k);
    r[4 * q + 3] = (w[q] >> 1) & 0x44444444u;
  }
}
// An operand row to this thread's lane of a slot (tmem = its columns at this warp's lanes).
__device__ __forceinline__ void operand_store(uint32_t tmem, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15,%16};" ::"r"(tmem),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void wait_stores() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Descriptor of a matrix at shared address a: leading (K) step 128 B, stride (row block) 512 B.
__device__ __forceinline__ uint64_t matrix_desc(uint32_t a) {
  return (uint64_t)((a >> 4) & 0x3fffu) | ((uint64_t)(128 >> 4) << 16) |
         ((uint64_t)(512 >> 4) << 32) | (1ull << 46);
}
// A and B e2m1, both K-major, e8m0 scales, N = 64, M = 128.
constexpr uint32_t kInstr = (1u << 7) | (1u << 10) | ((64u >> 3) << 17) | (1u << 23) |
                            ((128u >> 4) << 24);

// One instruction: 64 K positions of a slot times 64 rows.  A (converged) warp calls it and one
// lane issues.  All arguments are warp-uniform.
__device__ __forceinline__ void mma_step(uint32_t sums, uint32_t operand, uint64_t desc,
                                         uint32_t consts, uint32_t row_scales,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, z;\n"
      "elect.sync _|p, 0xffffffff;\nsetp.ne.u32 z, %6, 0;\n"
      "@p tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%4], "
      "[%5], z;\n}" ::"r"(sums),
      "r"(operand), "l"(desc), "r"(kInstr), "r"(consts), "r"(row_scales), "r"(accumulate)
      : "memory");
}
// The 2^11 that every sum starts from.
__device__ __forceinline__ void issue_ones(uint32_t sums, uint32_t consts, uint32_t ones) {
  mma_step(sums, consts + 12, matrix_desc(ones), consts, consts + 8, 0);
}
// The ones and a slot's products, all 128 output bits, rows n and n + 8 together, and the arrival
// on bar when they are done: one election for the whole sequence.
__device__ __forceinline__ void issue_pairs(uint32_t sums, uint32_t operand, uint32_t matrix,
                                            uint32_t consts, uint32_t ones, uint64_t* bar) {
  asm volatile(
      "{\n.reg .pred p, z, o;\n.reg .b64 l1, h0, h1;\n.reg .b32 a1, ones, s0, s1, s2;\n"
      "elect.sync _|p, 0xffffffff;\nsetp.ne.u32 z, 0, 0;\nsetp.eq.u32 o, 0, 0;\n"
      "add.u64 l1, %2, 16;\nadd.u64 h0, %2, %7;\nadd.u64 h1, %2, %8;\nadd.u32 a1, %1, 8;\n"
      "add.u32 ones, %4, 12;\nadd.u32 s0, %4, 8;\nadd.u32 s1, %4, 4;\nadd.u32 s2, %4, 6;\n"
      "@p tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [ones], %5, %3, [%4], "
      "[s0], z;\n"
      "@p tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%4], "
      "[s1], o;\n"
      "@p tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [a1], l1, %3, [%4], "
      "[s1], o;\n"
      "@p tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], h0, %3, [%4], "
      "[s2], o;\n"
      "@p tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [a1], h1, %3, [%4], "
      "[s2], o;\n"
      "@p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n}" ::"r"(
          sums),
      "r"(operand), "l"(matrix_desc(matrix)), "r"(kInstr), "r"(consts), "l"(matrix_desc(ones)),
      "r"(smem_addr(bar)), "n"(kMatrixBytes / 2 / 16), "n"(kMatrixBytes / 2 / 16 + 16)
      : "memory");
}
// A slot's products for the rows n with n / 8 mod 2 = part, one row to a sum.
__device__ __forceinline__ void issue_part(uint32_t sums, uint32_t operand, uint32_t matrix,
                                           uint32_t part, uint32_t consts) {
  const uint64_t desc = matrix_desc(matrix + part * (kMatrixBytes / 2));
  mma_step(sums, operand, desc, consts, consts + 4, 1);
  mma_step(sums, operand + 8, desc + 16, consts, consts + 4, 1);
}
// Arrives on bar when everything the warp issued is done.
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile(
      "{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\n"
      "@p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(
          smem_addr(bar))
      : "memory");
}

// The end of a launch, by the whole block: frees the tensor memory that its first warp allocated.
// When a wait of the block ran out, products may still be under way: every warp first waits (a
// bounded time) for what it issued, on a barrier of as many arrivals as the block has warps, and
// the launch is reported.
__device__ __forceinline__ void finish_launch(bool ok, uint64_t* drain, uint32_t tmem,
                                              uint32_t cols, uint32_t* stall_word) {
  fence_before();
  if (!__syncthreads_and(ok)) {
    commit(drain);
    bool drained = true;
    mbar_wait(drain, 0, drained);
    if (threadIdx.x == 0) report_stall(stall_word);
    __syncthreads();
  }
  if (threadIdx.x < 32) tmem_free(tmem, cols);
}

__device__ __forceinline__ void load_sums32(uint32_t tmem, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(tmem));
}
__device__ __forceinline__ void wait_loads() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Bits of a where mask has them, of b elsewhere.
__device__ __forceinline__ uint32_t take(uint32_t mask, uint32_t a, uint32_t b) {
  return (a & mask) | (b & ~mask);
}
// Bits j and j + 8 (field = 0x0101), or bit j (field = 0x01), of word j for j < 8; the other bits
// of the result mean nothing.
__device__ __forceinline__ uint32_t gather8(const uint32_t* s, uint32_t field) {
  const uint32_t a = take(field, s[0], s[1]), b = take(field << 2, s[2], s[3]);
  const uint32_t c = take(field << 4, s[4], s[5]), d = take(field << 6, s[6], s[7]);
  return take(field * 15, take(field * 3, a, b), take(field * 48, c, d));
}
// This thread's product from the sums of issue_pairs (tmem = their columns at this warp's lanes).
__device__ __forceinline__ uint4 collect_pairs(uint32_t tmem) {
  uint32_t r[32], o[4];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    load_sums32(tmem + 32 * h, r);
    wait_loads();
#pragma unroll
    for (int q = 0; q < 2; q++)
      o[2 * h + q] = __byte_perm(gather8(r + 16 * q, 0x0101u), gather8(r + 16 * q + 8, 0x0101u),
                                 0x5410);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
// Bytes 0 and 2 of each word of the product from part 0's sums, bytes 1 and 3 from part 1's: as
// eight bytes, those of words 0 and 1 in .x and of words 2 and 3 in .y.
__device__ __forceinline__ uint2 collect_part(uint32_t tmem) {
  uint32_t r[32], o[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    load_sums32(tmem + 32 * h, r);
    wait_loads();
    const uint32_t lo = __byte_perm(gather8(r, 1u), gather8(r + 8, 1u), 0x0040);
    const uint32_t hi = __byte_perm(gather8(r + 16, 1u), gather8(r + 24, 1u), 0x0040);
    o[h] = __byte_perm(lo, hi, 0x5410);
  }
  return make_uint2(o[0], o[1]);
}
__device__ __forceinline__ uint4 join_parts(uint2 p0, uint2 p1) {
  return make_uint4(__byte_perm(p0.x, p1.x, 0x5140), __byte_perm(p0.x, p1.x, 0x7362),
                    __byte_perm(p0.y, p1.y, 0x5140), __byte_perm(p0.y, p1.y, 0x7362));
}

}  // namespace tc
}  // namespace bgpu
