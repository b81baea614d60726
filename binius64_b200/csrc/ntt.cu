// Additive NTT (LCH14 "neighbors-last" form) and Reed-Solomon encode over GF(2^128).
//
// Semantics follow NeighborsLastReference (verifier/math/src/ntt/reference.rs:20-76): layer l acts
// on index bit (log_d - l - 1); block = idx >> (log_d - l) selects twiddle(l, block) =
// expanded[l][block] (GenericPreExpanded, ntt/domain_context.rs:99-159); the forward butterfly is
// u += v*t; v += u.  Field arithmetic is exact, so any evaluation order gives identical bits.
//
// B200 mapping: a pass fuses up to 13 consecutive layers.  One CTA owns a tile of 2^(k+c) elements
// (k butterfly bits plus c contiguous low index bits for coalescing) resident in shared memory
// together with the twiddles the tile needs, so each pass reads and writes HBM once with 128-bit
// accesses.  Transforms of 2^11 elements and more (but for narrow ranges of layers, tc_tile_bits)
// multiply on the tensor cores (ntt_tc_pass_kernel), others on the integer pipes (ntt_pass_kernel,
// up to 8 layers).  Reed-Solomon encode (reed_solomon.rs:128-201) fuses the message bit reversal
// and the 2^R-fold replication into the first pass's load: for the first pass the butterfly bits
// are exactly the message's low index bits after reversal, so the gather stays coalesced.
#include <algorithm>
#include <vector>

#include "gf128.cuh"
#include "gf_tc.cuh"
#include "internal.h"
#include "pdl.cuh"

using namespace bgpu;

namespace {

constexpr int kNttThreads = 256;
constexpr uint32_t kTileBits = 12;  // the largest tile: 4096 elements = 64 KiB of shared memory
constexpr uint32_t kMaxPassLayers = 8;

struct NttPass {
  uint32_t log_d;    // index bits of the whole buffer
  uint32_t l0;       // first layer of the pass
  uint32_t k;        // layers in the pass
  uint32_t c;        // contiguous low index bits in a tile
  uint32_t rs_bits;  // RS load: message index bits (bit-reversal width)
};

__device__ __forceinline__ uint32_t rev_bits32(uint32_t x, uint32_t n) {
  return n ? (__brev(x) >> (32 - n)) : 0u;
}
__device__ __forceinline__ uint64_t rev_bits64(uint64_t x, uint32_t n) {
  return n ? (__brevll(x) >> (64 - n)) : 0ull;
}

// twiddle(layer, j) = XOR of row[log_domain-1-layer][k+1] over the set bits k of j.
__global__ void expand_twiddles_kernel(uint4* __restrict__ tw, const uint4* __restrict__ rows,
                                       const uint32_t* __restrict__ row_offsets,
                                       uint32_t log_domain, uint64_t total) {
  for (uint64_t idx = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t layer = 63 - __clzll(idx + 1);
    uint64_t j = idx + 1 - (1ull << layer);
    const uint4* r = rows + row_offsets[log_domain - 1 - layer];
    uint4 acc = gf_zero();
    for (uint32_t k = 0; k < layer; k++)
      if ((j >> k) & 1) gf_add_into(acc, r[k + 1]);
    tw[idx] = acc;
  }
}

template <bool INVERSE, bool RS>
__global__ void __launch_bounds__(kNttThreads)
    ntt_pass_kernel(uint4* __restrict__ data, const uint4* __restrict__ src,
                    const uint4* __restrict__ tw, NttPass p) {
  pdl_wait();
  extern __shared__ uint4 smem[];
  const uint32_t k = p.k, c = p.c;
  const uint32_t tile_elems = 1u << (k + c);
  uint4* tile = smem;
  uint4* twl = smem + tile_elems;
  const uint32_t s = p.log_d - p.l0 - k;  // lowest butterfly index bit
  const uint64_t t = blockIdx.x;
  const uint64_t outer_mid = t & ((1ull << (s - c)) - 1);
  const uint64_t outer_hi = t >> (s - c);
  const uint64_t base = (outer_hi << (s + k)) | (outer_mid << c);

  // Twiddles of this tile: layer l0+m uses blocks (outer_hi << m) + [0, 2^m).
  for (uint32_t i = threadIdx.x; i + 1 < (1u << k); i += blockDim.x) {
    uint32_t m = 31 - __clz(i + 1);
    uint32_t j = i + 1 - (1u << m);
    uint64_t layer = p.l0 + m;
    twl[i] = __ldg(tw + ((1ull << layer) - 1) + (outer_hi << m) + j);
  }
  if (RS) {
    const uint64_t msg_mask = (p.rs_bits == 64) ? ~0ull : ((1ull << p.rs_bits) - 1);
    for (uint32_t e2 = threadIdx.x; e2 < tile_elems; e2 += blockDim.x) {
      uint32_t bfly = rev_bits32(e2 & ((1u << k) - 1), k);
      uint32_t inner = e2 >> k;
      uint64_t g = base | ((uint64_t)bfly << s) | inner;
      uint64_t si = rev_bits64(g & msg_mask, p.rs_bits);
      tile[(bfly << c) | inner] = __ldg(src + si);
    }
  } else {
    for (uint32_t e = threadIdx.x; e < tile_elems; e += blockDim.x) {
      uint64_t g = base | ((uint64_t)(e >> c) << s) | (e & ((1u << c) - 1));
      tile[e] = data[g];
    }
  }
  __syncthreads();

  const uint32_t half = tile_elems >> 1;
  for (uint32_t mm = 0; mm < k; mm++) {
    const uint32_t m = INVERSE ? (k - 1 - mm) : mm;
    const uint32_t h = c + k - 1 - m;
    for (uint32_t q = threadIdx.x; q < half; q += blockDim.x) {
      uint32_t e0 = ((q >> h) << (h + 1)) | (q & ((1u << h) - 1));
      uint32_t e1 = e0 | (1u << h);
      uint4 twd = twl[(1u << m) - 1 + (e0 >> (c + k - m))];
      uint4 u = tile[e0], v = tile[e1];
      if (!INVERSE) {
        gf_add_into(u, gf_mul(v, twd));
        gf_add_into(v, u);
      } else {
        gf_add_into(v, u);
        gf_add_into(u, gf_mul(v, twd));
      }
      tile[e0] = u;
      tile[e1] = v;
    }
    __syncthreads();
  }

  for (uint32_t e = threadIdx.x; e < tile_elems; e += blockDim.x) {
    uint64_t g = base | ((uint64_t)(e >> c) << s) | (e & ((1u << c) - 1));
    data[g] = tile[e];
  }
}

// ---- the tensor-core pass
//
// The same pass on a tile of 2^10 to 2^13 elements (up to 128 KiB of shared memory), one CTA of
// four 128-thread groups per SM, persistent over the tiles.  A layer's butterflies are taken 128 at a time (an M-tile),
// v t by gf_tc.cuh; a group has a contiguous share of the layer's M-tiles, and prepares the next
// one while the tensor cores work on this:
//
// * butterfly bit h >= 7: an M-tile has one twiddle.  Its matrix is built when it changes, under
//   the products of the M-tile before.
// * h = 6, 5: two or four twiddles.  They differ by the layer's twiddles of blocks 1 and 2
//   (twiddle(block) is linear in the block's bits), whose matrices are built once per layer; the
//   M-tile's own matrix is the one of its first twiddle, and each row bit from h up is an operand
//   slot.  Measured per layer of a 2^13 tile: 25 and 28 k cycles, against 34 k with the integer
//   multiply and 14 k with one twiddle; with four and five slots (h = 4, 3) 31 and 34 k.
// * h < 5: the integer multiply.
//
// What bounds it (five and four layers of a 2^13-element tile, ncu): the logic pipe 63% and the
// tensor pipe 40% busy with 16 warps an SM, DRAM 12%.  Per 128 products and one layer 450 cycles,
// of which a lone stream of collections and operand writes takes 235 (tensor-memory reads do not
// overlap the logic that follows them); the rest is the hand-over between a group's warps (four of
// them must have read the sums before the next products start, and four groups are all that 512
// TMEM columns hold with two operand slots each), a fifth of it the drain at the end of a layer.
// Measured against it and left: three groups with 128 columns of sums and e4m3 / e5m2 operands
// (690 cycles per 128 products and layer), a separate issuing warp that polls the groups (750).
constexpr uint32_t kTcGroups = 4;
constexpr uint32_t kTcThreads = kTcGroups * tc::kGroupThreads;
constexpr uint32_t kTcTileBits = 13;
constexpr uint32_t kTcMinTileBits = 10;
constexpr uint32_t kTcOneBit = 7;     // an M-tile has one twiddle from this butterfly bit up
constexpr uint32_t kTcLowestBit = 5;  // and takes slots down to this one
constexpr uint32_t kTcLowLayers = kTcOneBit - kTcLowestBit;
constexpr uint32_t kTcTmemCols = 512;
constexpr uint32_t kTcMaxMTiles = 1u << (kTcTileBits - 8);
constexpr uint32_t kTcLowTwiddles = kTcMaxMTiles + kTcLowLayers;  // of one layer with h < 7
constexpr uint32_t kTcTwiddles = 2 * kTcMaxMTiles + kTcLowLayers * kTcLowTwiddles;
constexpr uint32_t kTcMatrices = 2 * kTcGroups;

struct NttTcShared {
  uint4 tile[1u << kTcTileBits];
  uint8_t matrices[kTcMatrices][tc::kMatrixBytes];
  tc::MatrixRows rows[2][kTcLowTwiddles];  // of this layer's and the next one's twiddles
  uint4 twiddles[kTcTwiddles];
  uint8_t ones[tc::kOnesBytes];
  uint64_t done[kTcGroups], drain;
  uint32_t tmem;
};

__device__ __forceinline__ void cp_async16(uint4* smem_dst, const uint4* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_addr(smem_dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// One layer of a tile in shared memory on the tensor cores (SLOTS: h < 7); emit(e, x) takes the
// results.  `ok` becomes false when a wait runs out.
template <bool INVERSE, bool SLOTS, class Emit>
__device__ __forceinline__ void ntt_tc_layer(NttTcShared& sh, const tc::MatrixRows* rows,
                                             uint32_t h, uint32_t n_mtiles, uint32_t group,
                                             uint32_t tmem, uint32_t& phase, bool& ok,
                                             const Emit& emit) {
  const uint32_t gt = threadIdx.x % tc::kGroupThreads;
  const uint32_t gw = tc::uniform(gt / 32);
  const uint32_t lanes = (gw * 32) << 16;
  const uint32_t row_bits = SLOTS ? kTcOneBit - h : 0;
  // TMEM columns of a group: its sums, then two operand slots in turn, or the M-tile's slots
  constexpr uint32_t cols = tc::kSumCols + tc::kOperandCols * (1 + kTcLowLayers);
  static_assert(kTcGroups * cols + tc::kConstCols <= kTcTmemCols, "TMEM columns");
  const uint32_t sums = tmem + group * cols;
  const uint32_t slot0 = sums + tc::kSumCols;
  const uint32_t consts = tmem + kTcTmemCols - tc::kConstCols;
  const uint32_t ones = tc::uniform(tc::smem_addr(sh.ones));
  const uint32_t matrices = tc::uniform(tc::smem_addr(sh.matrices));
  uint32_t buf = SLOTS ? group : 2 * group;

  if (SLOTS) {  // the matrices of the layer's twiddles of blocks 1, 2, 4, ..
    if (group < row_bits) {
      tc::matrix_build(sh.matrices[kTcGroups + group], rows[n_mtiles + group], gt);
      tc::fence_smem_to_tensor();
    }
    __syncthreads();
  }
  const uint32_t i0 = n_mtiles * group / kTcGroups, i1 = n_mtiles * (group + 1) / kTcGroups;

  const uint32_t hs = SLOTS ? 0 : h - kTcOneBit;  // M-tile i has twiddle i >> hs
  auto first = [&](uint32_t i) {  // the tile index of this thread's u
    if (SLOTS) {
      const uint32_t q = i * tc::kGroupThreads + gt;
      return ((q >> h) << (h + 1)) | (q & ((1u << h) - 1));
    }
    return ((i >> hs) << (h + 1)) + ((i & ((1u << hs) - 1)) * tc::kGroupThreads) + gt;
  };
  auto build = [&](uint32_t j) {
    tc::matrix_build(sh.matrices[buf], rows[j], gt);
    tc::fence_smem_to_tensor();
  };
  uint32_t slot = slot0;
  auto store_operand = [&](uint4 x) {
    uint32_t r[16];
    tc::operand_words(x, r);
    tc::operand_store(slot + lanes, r);
    if (SLOTS) {
      for (uint32_t j = 0; j < row_bits; j++) {
        const bool on = (gt >> (h + j)) & 1;
        uint32_t m[16];
#pragma unroll
        for (int w = 0; w < 16; w++) m[w] = on ? r[w] : 0u;
        tc::operand_store(slot0 + tc::kOperandCols * (1 + j) + lanes, m);
      }
    }
    tc::wait_stores();
  };
  // operand and matrix written, sums read by the whole group: one warp issues the next products
  auto start = [&](uint32_t turn, uint32_t part) {
    tc::fence_before();
    if (gw != (turn & 3)) {
      tc::group_arrive(group + 1);
      return;
    }
    tc::group_wait(group + 1);
    tc::fence_after();
    if (!SLOTS) {
      tc::issue_pairs(sums, slot, matrices + buf * tc::kMatrixBytes, consts, ones,
                      &sh.done[group]);
      return;
    }
    tc::issue_ones(sums, consts, ones);
    tc::issue_part(sums, slot, matrices + buf * tc::kMatrixBytes, part, consts);
    for (uint32_t j = 0; j < row_bits; j++)
      tc::issue_part(sums, slot0 + tc::kOperandCols * (1 + j),
                     matrices + (kTcGroups + j) * tc::kMatrixBytes, part, consts);
    tc::commit(&sh.done[group]);
  };
  auto finish = [&]() {
    tc::mbar_wait(&sh.done[group], phase, ok);
    phase ^= 1;
    tc::fence_after();
  };

  build(i0 >> hs);
  uint32_t e0 = first(i0);
  uint4 u = sh.tile[e0], v = sh.tile[e0 | (1u << h)];
  if (INVERSE) gf_add_into(v, u);
  store_operand(v);
  start(i0, 0);
  for (uint32_t i = i0; i < i1; i++) {
    const bool next = i + 1 < i1;
    uint32_t ne0 = e0;
    uint4 nu = u, nv = v, tv;
    uint2 part0;
    if (SLOTS) {
      finish();
      part0 = tc::collect_part(sums + lanes);
      start(i + 1, 1);
    }
    if (next) {
      ne0 = first(i + 1);
      nu = sh.tile[ne0];
      nv = sh.tile[ne0 | (1u << h)];
      if (INVERSE) gf_add_into(nv, nu);
      if (!SLOTS) {
        if (((i + 1) >> hs) != (i >> hs)) {
          buf ^= 1;
          build((i + 1) >> hs);
        }
        slot ^= slot0 ^ (slot0 + tc::kOperandCols);
        store_operand(nv);
      }
    }
    finish();
    if (SLOTS) {
      if (next) {
        build(i + 1);
        store_operand(nv);
      }
      tv = tc::join_parts(part0, tc::collect_part(sums + lanes));
    } else {
      tv = tc::collect_pairs(sums + lanes);
    }
    if (next) start(i + 1, 0);
    gf_add_into(u, tv);
    if (!INVERSE) gf_add_into(v, u);
    emit(e0, u);
    emit(e0 | (1u << h), v);
    e0 = ne0;
    u = nu;
    v = nv;
  }
}

template <bool INVERSE, bool RS>
__global__ void __launch_bounds__(kTcThreads, 1)
    ntt_tc_pass_kernel(uint4* __restrict__ data, const uint4* __restrict__ src,
                       const uint4* __restrict__ tw, NttPass p, uint32_t n_tiles,
                       uint32_t* stall_word) {
  pdl_wait();
  extern __shared__ __align__(128) uint8_t tc_smem[];
  NttTcShared& sh = *reinterpret_cast<NttTcShared*>(tc_smem);
  const uint32_t k = p.k, c = p.c;
  const uint32_t tile_elems = 1u << (k + c);
  const uint32_t s = p.log_d - p.l0 - k;  // lowest butterfly index bit
  const uint32_t half = tile_elems >> 1;
  const uint32_t n_mtiles = half / tc::kGroupThreads;
  const uint32_t n_one = min(k, c + k - kTcOneBit);           // layers with h >= kTcOneBit
  const uint32_t n_low = min(k - n_one, kTcLowLayers);        // with kTcOneBit > h >= kTcLowestBit
  const uint32_t group = tc::uniform(threadIdx.x / tc::kGroupThreads);

  // element e of a tile <-> its base | e's butterfly bits << s | its low c bits
  auto tile_base = [&](uint32_t t) {
    return ((uint64_t)(t >> (s - c)) << (s + k)) | ((uint64_t)(t & ((1u << (s - c)) - 1)) << c);
  };
  auto tile_offset = [&](uint32_t e) { return ((uint64_t)(e >> c) << s) | (e & ((1u << c) - 1)); };
  auto load_tile = [&](uint32_t t) {
    const uint64_t base = tile_base(t);
    for (uint32_t e = threadIdx.x; e < tile_elems; e += kTcThreads) {
      if (RS) {
        const uint64_t msg_mask = (p.rs_bits == 64) ? ~0ull : ((1ull << p.rs_bits) - 1);
        const uint32_t bfly = rev_bits32(e & ((1u << k) - 1), k);
        const uint32_t inner = e >> k;
        const uint64_t g = base | ((uint64_t)bfly << s) | inner;
        cp_async16(sh.tile + ((bfly << c) | inner), src + rev_bits64(g & msg_mask, p.rs_bits));
      } else {
        cp_async16(sh.tile + e, data + (base | tile_offset(e)));
      }
    }
  };
  // its twiddles: layer l0 + m uses blocks (outer_hi << m) + [0, 2^m).  Layers with h >= 7 keep
  // them all (at 2^m - 1); one below keeps each M-tile's first and those of blocks 1, 2, 4, ..
  auto load_twiddles = [&](uint32_t t) {
    const uint64_t outer_hi = (uint64_t)t >> (s - c);
    for (uint32_t i = threadIdx.x; i + 1 < (1u << n_one); i += kTcThreads) {
      const uint32_t m = 31 - __clz(i + 1);
      cp_async16(sh.twiddles + i,
                 tw + ((1ull << (p.l0 + m)) - 1) + (outer_hi << m) + (i + 1 - (1u << m)));
    }
    for (uint32_t x = threadIdx.x; x < n_low * kTcLowTwiddles; x += kTcThreads) {
      const uint32_t low = x / kTcLowTwiddles, i = x % kTcLowTwiddles, m = n_one + low;
      const uint4* layer = tw + ((1ull << (p.l0 + m)) - 1);
      uint4* dst = sh.twiddles + 2 * kTcMaxMTiles + low * kTcLowTwiddles + i;
      if (i < n_mtiles)
        cp_async16(dst, layer + (outer_hi << m) + ((uint64_t)i << (low + 1)));
      else if (i < n_mtiles + low + 1)
        cp_async16(dst, layer + (1u << (i - n_mtiles)));
    }
  };
  // the matrix rows of layer m's twiddles into the buffer of its parity
  auto prepare_rows = [&](uint32_t m) {
    if (m >= n_one + n_low) return;
    const bool one = m < n_one;
    const uint4* t = sh.twiddles + (one ? (1u << m) - 1
                                        : 2 * kTcMaxMTiles + (m - n_one) * kTcLowTwiddles);
    const uint32_t n = one ? 1u << m : n_mtiles + m - n_one + 1;
    for (uint32_t x = threadIdx.x; x < n * tc::kRowItems; x += kTcThreads)
      tc::matrix_rows(sh.rows[m & 1][x / tc::kRowItems], t[x / tc::kRowItems], x % tc::kRowItems);
  };

  if (threadIdx.x < 32) tc::tmem_alloc(&sh.tmem, kTcTmemCols);
  if (threadIdx.x == 0) {
    for (uint32_t g = 0; g < kTcGroups; g++) tc::mbar_init(&sh.done[g], 1);
    tc::mbar_init(&sh.drain, kTcThreads / 32);
    tc::mbar_init_fence();
  }
  load_tile(blockIdx.x);
  load_twiddles(blockIdx.x);
  cp_async_wait_all();
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tc::uniform(sh.tmem);
  if (group == 0) {
    tc::constants_store(tmem + kTcTmemCols - tc::kConstCols + ((threadIdx.x / 32 * 32) << 16),
                        sh.ones);
    tc::fence_smem_to_tensor();
  }
  prepare_rows(INVERSE ? k - 1 : 0);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();

  uint32_t phase = 0;
  bool ok = true;
  for (uint32_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    const uint64_t outer_hi = (uint64_t)t >> (s - c);
    const uint32_t nt = t + gridDim.x;
    uint4* out = data + tile_base(t);
    const uint4* next = data + (nt < n_tiles ? tile_base(nt) : 0);
    for (uint32_t mm = 0; mm < k; mm++) {
      const uint32_t m = INVERSE ? (k - 1 - mm) : mm;
      const uint32_t h = c + k - 1 - m;
      const bool last = mm + 1 == k;
      // The last layer's results go to memory at once, and the next tile's elements come into the
      // places that are now free.
      auto emit = [&](uint32_t e, uint4 x) {
        if (!last) {
          sh.tile[e] = x;
          return;
        }
        const uint64_t offset = tile_offset(e);
        out[offset] = x;
        if (!RS && nt < n_tiles) cp_async16(sh.tile + e, next + offset);
      };
      const tc::MatrixRows* rows = sh.rows[m & 1];
      if (h >= kTcOneBit) {
        ntt_tc_layer<INVERSE, false>(sh, rows, h, n_mtiles, group, tmem, phase, ok, emit);
      } else if (h >= kTcLowestBit) {
        ntt_tc_layer<INVERSE, true>(sh, rows, h, n_mtiles, group, tmem, phase, ok, emit);
      } else {
        const uint4* lt = tw + ((1ull << (p.l0 + m)) - 1) + (outer_hi << m);
        for (uint32_t q = threadIdx.x; q < half; q += kTcThreads) {
          const uint32_t e0 = ((q >> h) << (h + 1)) | (q & ((1u << h) - 1));
          const uint32_t e1 = e0 | (1u << h);
          const uint4 twd = __ldg(lt + (q >> h));
          uint4 u = sh.tile[e0], v = sh.tile[e1];
          if (!INVERSE) {
            gf_add_into(u, gf_mul(v, twd));
            gf_add_into(v, u);
          } else {
            gf_add_into(v, u);
            gf_add_into(u, gf_mul(v, twd));
          }
          emit(e0, u);
          emit(e1, v);
        }
      }
      if (!last) {
        prepare_rows(INVERSE ? m - 1 : m + 1);
        __syncthreads();
      }
    }
    if (nt < n_tiles) {
      __syncthreads();
      if (RS) load_tile(nt);
      load_twiddles(nt);
      cp_async_wait_all();
      __syncthreads();
      prepare_rows(INVERSE ? k - 1 : 0);
      __syncthreads();
    }
  }
  tc::finish_launch(ok, &sh.drain, tmem, kTcTmemCols, stall_word);
}

std::vector<NttPass> plan_passes(uint32_t log_d, uint32_t skip_early, uint32_t skip_late,
                                 bool rs, uint32_t rs_bits) {
  // tiles of 2^tile_bits elements: fewer, larger tiles fuse more work per CTA; more, smaller ones
  // spread a small transform evenly over the 148 SMs (a 2^20 codeword is 256 tiles of 2^12)
  const uint32_t tile_bits = std::max(9u, std::min(kTileBits, tuning().ntt_tile_bits));
  std::vector<NttPass> passes;
  uint32_t n_layers = log_d - skip_late - skip_early;
  if (n_layers == 0) {
    if (rs) {
      uint32_t s = log_d - skip_early;
      passes.push_back({log_d, skip_early, 0, std::min(tile_bits, s), rs_bits});
    }
    return passes;
  }
  const uint32_t max_layers =
      std::max(1u, std::min({kMaxPassLayers, tuning().ntt_pass_layers, tile_bits}));
  uint32_t n_passes = (n_layers + max_layers - 1) / max_layers;
  uint32_t base = n_layers / n_passes, extra = n_layers % n_passes;
  uint32_t l0 = skip_early;
  for (uint32_t i = 0; i < n_passes; i++) {
    uint32_t k = base + (i < extra ? 1 : 0);
    uint32_t s = log_d - l0 - k;
    uint32_t c = std::min(tile_bits - k, s);
    passes.push_back({log_d, l0, k, c, i == 0 ? rs_bits : 0u});
    l0 += k;
  }
  return passes;
}

// The tensor-core passes of a transform: tiles of 2^tile_bits elements.  The last pass takes every
// layer its tile can hold above the skipped low bits (its layers below bit 7 are the slower ones
// whatever the split); the others keep at least 2^7 contiguous elements, so that each M-tile of
// theirs has one twiddle, and are as even as they can be.
std::vector<NttPass> plan_tc_passes(uint32_t log_d, uint32_t skip_early, uint32_t skip_late,
                                    uint32_t tile_bits, uint32_t rs_bits) {
  std::vector<NttPass> passes;
  const uint32_t n_layers = log_d - skip_late - skip_early;
  const uint32_t most = tile_bits - kTcOneBit;
  const uint32_t last = std::min(n_layers, tile_bits - std::min(skip_late, kTcOneBit));
  const uint32_t rest = n_layers - last;
  const uint32_t n_rest = (rest + most - 1) / most;
  uint32_t l0 = skip_early;
  for (uint32_t i = 0; i <= n_rest; i++) {
    const uint32_t k = i == n_rest ? last : rest / n_rest + (i < rest % n_rest ? 1 : 0);
    const uint32_t s = log_d - l0 - k;
    passes.push_back({log_d, l0, k, std::min(tile_bits - k, s), i == 0 ? rs_bits : 0u});
    l0 += k;
  }
  return passes;
}

// Tile bits of a transform's tensor-core passes, 0 = the integer passes.  2^(log_d - 7) elements
// a tile gives 128 CTAs for the 148 SMs; beyond 2^20 the largest tile that fits (fewer passes and
// fewer matrices per product), below 2^17 the smallest whose four groups all have an M-tile.
// Measured on B200, Reed-Solomon encode / inverse transform in us, integer passes -> these:
// 2^26 x 64 columns 17320 -> 7690, 2^24 x 16 4399 -> 2190, 2^20 x 16 265 -> 134 (tiles of 2^12:
// 157), 2^18 x 16 99 -> 53 (2^12: 72, 2^10: 74), 2^16 x 16 70 -> 37, 2^12 x 16 36 -> 25; inverse
// 2^22 .. 2^12 at 0.5-0.6 of the time.
//
// Where the butterflies stay within ten index bits (log_d - skip_early = 10, one pass of one layer a
// bit) and up to 32 tiles of them, the integer passes are at least as fast: they spread such a tile
// over more CTAs.  Integer against tensor-core passes, in us: 2^11 elements without the first layer
// 19.0 and 25.7 (encodes at rate 1/2 19.2 and 25.8, 2^12 at rate 1/4 19.4 and 25.9), and without
// the last two 20.6 and 21.0; 2^15 without the first five 24.2 and 25.9; 2^16 without the first six
// 33.8 and 26.0.  With eleven bits they lose: 2^11 35.4 and 30.0, 2^12 without the first layer 35.1
// and 29.8, 2^15 without the first four 40.4 and 30.1.
uint32_t tc_tile_bits(uint32_t log_d, uint32_t skip_early, uint32_t skip_late) {
  if (log_d == skip_early + skip_late) return 0;
  if (log_d < 16 && log_d - skip_early <= kTcMinTileBits) return 0;
  const uint32_t bits = std::min(std::max(log_d - 7, kTcMinTileBits), kTcTileBits);
  return log_d - skip_early >= bits ? bits : 0;
}

template <bool INVERSE, bool RS>
int launch_tc_pass(const NttPass& p, uint4* data, const uint4* src, const uint4* tw,
                   cudaStream_t stream) {
  auto kern = ntt_tc_pass_kernel<INVERSE, RS>;
  if (int rc = ensure_smem_limit(reinterpret_cast<const void*>(kern), sizeof(NttTcShared))) return rc;
  const uint64_t n_tiles = 1ull << (p.log_d - p.k - p.c);
  if (n_tiles > 0x7fffffffull) return set_error(BINIUS_E_ARG, "ntt: buffer too large");
  uint32_t* stall_word = nullptr;
  if (int rc = tensor_word(&stall_word)) return rc;
  launch_pdl(kern, (unsigned)std::min<uint64_t>(n_tiles, 148), kTcThreads, sizeof(NttTcShared),
             stream, data, src, tw, p, (uint32_t)n_tiles, stall_word);
  BGPU_LAUNCH_CHECK("ntt_tc_pass_kernel");
  count_launch();
  return BINIUS_OK;
}

template <bool INVERSE, bool RS>
int launch_pass(const NttPass& p, uint4* data, const uint4* src, const uint4* tw,
                cudaStream_t stream) {
  size_t smem = ((size_t(1) << (p.k + p.c)) + (size_t(1) << p.k) - 1) * sizeof(uint4);
  auto kern = ntt_pass_kernel<INVERSE, RS>;
  // the largest tile of any pass: 2^kTileBits elements plus 2^kMaxPassLayers - 1 twiddles
  constexpr size_t kMaxSmem = ((size_t(1) << kTileBits) + (size_t(1) << kMaxPassLayers) - 1) *
                              sizeof(uint4);
  if (smem > kMaxSmem) return set_error(BINIUS_E_ARG, "ntt: pass tile exceeds the planned maximum");
  if (int rc = ensure_smem_limit(reinterpret_cast<const void*>(kern), kMaxSmem)) return rc;
  uint64_t n_tiles = 1ull << (p.log_d - p.k - p.c);
  if (n_tiles > 0x7fffffffull) return set_error(BINIUS_E_ARG, "ntt: buffer too large");
  launch_pdl(kern, (unsigned)n_tiles, kNttThreads, smem, stream, data, src, tw, p);
  BGPU_LAUNCH_CHECK("ntt_pass_kernel");
  count_launch();
  return BINIUS_OK;
}

int check_device(const binius_ntt* ntt) {
  int dev = -1;
  BGPU_CUDA(cudaGetDevice(&dev));
  if (dev != ntt->device)
    return set_error(BINIUS_E_ARG, "binius_ntt used on a device other than the one it was built on");
  return BINIUS_OK;
}

int ntt_transform(const binius_ntt* ntt, void* d_data, uint32_t log_len, uint32_t skip_early,
                  uint32_t skip_late, void* stream, bool inverse) {
  BGPU_ARG(ntt != nullptr, "ntt is NULL");
  BGPU_ARG(d_data != nullptr || log_len == 0, "data is NULL");
  BGPU_ARG(log_len <= 40, "log_len too large");
  // input_check (ntt/reference.rs:85-100)
  BGPU_ARG(skip_early + skip_late <= log_len, "skip_early + skip_late must be <= log_len");
  BGPU_ARG(log_len - skip_late <= ntt->log_domain, "domain context too small for the transform");
  if (int rc = check_device(ntt)) return rc;
  uint4* data = static_cast<uint4*>(d_data);
  const uint4* tw = static_cast<const uint4*>(ntt->d_twiddles);
  cudaStream_t s = as_stream(stream);
  if (const uint32_t tb = tc_tile_bits(log_len, skip_early, skip_late)) {
    auto passes = plan_tc_passes(log_len, skip_early, skip_late, tb, 0);
    if (!inverse) {
      for (const auto& p : passes)
        if (int rc = launch_tc_pass<false, false>(p, data, nullptr, tw, s)) return rc;
    } else {
      for (auto it = passes.rbegin(); it != passes.rend(); ++it)
        if (int rc = launch_tc_pass<true, false>(*it, data, nullptr, tw, s)) return rc;
    }
    return clear_error();
  }
  auto passes = plan_passes(log_len, skip_early, skip_late, false, 0);
  if (!inverse) {
    for (const auto& p : passes)
      if (int rc = launch_pass<false, false>(p, data, nullptr, tw, s)) return rc;
  } else {
    for (auto it = passes.rbegin(); it != passes.rend(); ++it)
      if (int rc = launch_pass<true, false>(*it, data, nullptr, tw, s)) return rc;
  }
  return clear_error();
}

}  // namespace

namespace bgpu {

bool rs_encode_is_tuned(uint32_t log_dim, uint32_t log_inv_rate, uint32_t log_batch) {
  return tc_tile_bits(log_dim + log_batch + log_inv_rate, log_inv_rate, log_batch) == 0;
}

int rs_encode_batch(const binius_ntt* ntt, const void* d_msg, uint32_t log_dim,
                    uint32_t log_inv_rate, uint32_t log_batch, void* d_codeword,
                    cudaStream_t stream) {
  BGPU_ARG(ntt != nullptr, "ntt is NULL");
  BGPU_ARG(d_msg != nullptr && d_codeword != nullptr, "msg / codeword is NULL");
  BGPU_ARG(d_msg != d_codeword, "codeword must not alias the message");
  uint32_t log_msg = log_dim + log_batch;
  uint32_t log_out = log_msg + log_inv_rate;
  BGPU_ARG(log_out <= 40, "codeword too large");
  // encode_batch requires the NTT subspace of dimension log_len (reed_solomon.rs:143-145)
  BGPU_ARG(log_dim + log_inv_rate <= ntt->log_domain,
           "NTT domain smaller than the code's evaluation domain");
  if (int rc = check_device(ntt)) return rc;
  uint4* out = static_cast<uint4*>(d_codeword);
  const uint4* msg = static_cast<const uint4*>(d_msg);
  const uint4* tw = static_cast<const uint4*>(ntt->d_twiddles);
  if (const uint32_t tb = tc_tile_bits(log_out, log_inv_rate, log_batch)) {
    auto passes = plan_tc_passes(log_out, log_inv_rate, log_batch, tb, log_msg);
    for (size_t i = 0; i < passes.size(); i++) {
      int rc = (i == 0) ? launch_tc_pass<false, true>(passes[i], out, msg, tw, stream)
                        : launch_tc_pass<false, false>(passes[i], out, nullptr, tw, stream);
      if (rc) return rc;
    }
    return clear_error();
  }
  auto passes = plan_passes(log_out, log_inv_rate, log_batch, true, log_msg);
  for (size_t i = 0; i < passes.size(); i++) {
    int rc = (i == 0) ? launch_pass<false, true>(passes[i], out, msg, tw, stream)
                      : launch_pass<false, false>(passes[i], out, nullptr, tw, stream);
    if (rc) return rc;
  }
  return clear_error();
}

}  // namespace bgpu

namespace {

// generate_evals_from_subspace (ntt/domain_context.rs:19-46): row i holds the normalized
// subspace-polynomial evaluations [W_i(b_i), W_i(b_(i+1)), ...] / W_i(b_i) of the domain basis
// (h_basis: l elements, or NULL for BinarySubspace::with_dim's basis x^i).
int subspace_evals(const void* h_basis, uint32_t l, std::vector<std::vector<hu128>>& evals) {
  std::vector<hu128> basis(l);
  for (uint32_t i = 0; i < l; i++) {
    if (h_basis) {
      const uint64_t* b = static_cast<const uint64_t*>(h_basis) + 2 * i;
      basis[i] = ((hu128)b[1] << 64) | b[0];
    } else {
      basis[i] = (hu128)1 << i;
    }
  }
  evals.clear();
  evals.push_back(basis);
  for (uint32_t i = 1; i < l; i++) {
    const auto& prev = evals[i - 1];
    std::vector<hu128> row;
    for (size_t k = 1; k < prev.size(); k++) row.push_back(host_gf_mul(prev[k], prev[k] ^ prev[0]));
    evals.push_back(row);
  }
  for (auto& row : evals) {
    if (row[0] == 0) return set_error(BINIUS_E_ARG, "subspace basis is linearly dependent");
    hu128 inv = host_gf_inv(row[0]);
    for (auto& v : row) v = host_gf_mul(v, inv);
  }
  return BINIUS_OK;
}

}  // namespace

extern "C" {

int binius_domain_subspace(const void* h_basis, uint32_t log_domain, uint32_t dim, void* h_out) {
  BGPU_ARG(h_out != nullptr, "out is NULL");
  BGPU_ARG(log_domain >= 1 && log_domain <= 64, "log_domain must be in [1, 64]");
  BGPU_ARG(dim <= log_domain, "dim must be <= log_domain");
  uint64_t* o = static_cast<uint64_t*>(h_out);
  if (dim == 0) return clear_error();  // BinarySubspace::with_dim(0)
  std::vector<std::vector<hu128>> evals;
  if (int rc = subspace_evals(h_basis, log_domain, evals)) return rc;
  const auto& row = evals[log_domain - dim];
  for (uint32_t i = 0; i < dim; i++) {
    o[2 * i] = (uint64_t)row[i];
    o[2 * i + 1] = (uint64_t)(row[i] >> 64);
  }
  return clear_error();
}

int binius_ntt_create(int device, const void* h_basis, uint32_t log_domain, binius_ntt** out) {
  BGPU_ARG(out != nullptr, "out is NULL");
  *out = nullptr;
  BGPU_ARG(log_domain >= 1 && log_domain <= 32, "log_domain must be in [1, 32]");
  if (int rc = configure_device_pool(device)) return rc;
  uint32_t* stall_word = nullptr;  // made here rather than by the first transform
  if (int rc = tensor_word(&stall_word)) return rc;
  const uint32_t l = log_domain;
  std::vector<std::vector<hu128>> evals;
  if (int rc = subspace_evals(h_basis, l, evals)) return rc;
  std::vector<uint32_t> offsets(l);
  std::vector<uint64_t> packed;
  for (uint32_t i = 0; i < l; i++) {
    offsets[i] = (uint32_t)(packed.size() / 2);
    for (hu128 v : evals[i]) {
      packed.push_back((uint64_t)v);
      packed.push_back((uint64_t)(v >> 64));
    }
  }

  int prev_dev = 0;
  BGPU_CUDA(cudaGetDevice(&prev_dev));
  BGPU_CUDA(cudaSetDevice(device));
  uint64_t total = (1ull << l) - 1;
  void* d_tw = nullptr;
  void* d_rows = nullptr;
  void* d_off = nullptr;
  int rc = BINIUS_OK;
  do {
    cudaError_t e = cudaMalloc(&d_tw, total * 16);
    if (e != cudaSuccess) { rc = cuda_error(e, "cudaMalloc(twiddles)"); break; }
    e = cudaMalloc(&d_rows, packed.size() * 8);
    if (e != cudaSuccess) { rc = cuda_error(e, "cudaMalloc(rows)"); break; }
    e = cudaMalloc(&d_off, offsets.size() * 4);
    if (e != cudaSuccess) { rc = cuda_error(e, "cudaMalloc(offsets)"); break; }
    e = cudaMemcpy(d_rows, packed.data(), packed.size() * 8, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) { rc = cuda_error(e, "cudaMemcpy(rows)"); break; }
    e = cudaMemcpy(d_off, offsets.data(), offsets.size() * 4, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) { rc = cuda_error(e, "cudaMemcpy(offsets)"); break; }
    unsigned blocks = (unsigned)std::min<uint64_t>((total + 255) / 256, 148ull * 32);
    expand_twiddles_kernel<<<blocks, 256>>>(static_cast<uint4*>(d_tw),
                                            static_cast<const uint4*>(d_rows),
                                            static_cast<const uint32_t*>(d_off), l, total);
    e = cudaGetLastError();
    if (e != cudaSuccess) { rc = cuda_error(e, "expand_twiddles_kernel"); break; }
    e = cudaDeviceSynchronize();
    if (e != cudaSuccess) { rc = cuda_error(e, "expand_twiddles_kernel sync"); break; }
  } while (0);
  if (d_rows) cudaFree(d_rows);
  if (d_off) cudaFree(d_off);
  if (rc != BINIUS_OK) {
    if (d_tw) cudaFree(d_tw);
    cudaSetDevice(prev_dev);
    return rc;
  }
  binius_ntt* ntt = new binius_ntt;
  ntt->device = device;
  ntt->log_domain = l;
  ntt->d_twiddles = d_tw;
  *out = ntt;
  cudaSetDevice(prev_dev);
  return clear_error();
}

int binius_ntt_destroy(binius_ntt* ntt) {
  if (!ntt) return BINIUS_OK;
  int prev_dev = 0;
  cudaGetDevice(&prev_dev);
  cudaSetDevice(ntt->device);
  cudaFree(ntt->d_twiddles);
  cudaSetDevice(prev_dev);
  delete ntt;
  return BINIUS_OK;
}

uint32_t binius_ntt_log_domain(const binius_ntt* ntt) { return ntt ? ntt->log_domain : 0; }

const void* binius_ntt_twiddles(const binius_ntt* ntt) { return ntt ? ntt->d_twiddles : nullptr; }

int binius_ntt_forward(const binius_ntt* ntt, void* d_data, uint32_t log_len, uint32_t skip_early,
                       uint32_t skip_late, void* stream) {
  return ntt_transform(ntt, d_data, log_len, skip_early, skip_late, stream, false);
}

int binius_ntt_inverse(const binius_ntt* ntt, void* d_data, uint32_t log_len, uint32_t skip_early,
                       uint32_t skip_late, void* stream) {
  return ntt_transform(ntt, d_data, log_len, skip_early, skip_late, stream, true);
}

int binius_rs_encode_batch(const binius_ntt* ntt, const void* d_msg, uint32_t log_dim,
                           uint32_t log_inv_rate, uint32_t log_batch, void* d_codeword,
                           void* stream) {
  return bgpu::rs_encode_batch(ntt, d_msg, log_dim, log_inv_rate, log_batch, d_codeword,
                               as_stream(stream));
}

}  // extern "C"
