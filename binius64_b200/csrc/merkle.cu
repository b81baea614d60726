// Binary Merkle tree commit with SHA-256 leaves and the Binius SHA-256 node compression.
//
// Layout follows BinaryMerkleTree::inner_nodes (prover/prover/src/merkle_tree/binary_merkle_tree.rs
// :65-122): 2^(L+1) - 1 digests of 32 bytes, the 2^L leaf digests first, then each layer, the root
// last; node i of layer k+1 compresses nodes 2i and 2i+1 of layer k (parallel_compression.rs:79-91).
//
// B200 mapping: one thread hashes one leaf (its 2^log_batch elements are read as 128-bit loads);
// the CTA's 256 leaf digests stay in shared memory and the next tree layers are compressed there
// before anything but the layer outputs touches HBM: all 8 of them in a tree of up to 2^16 leaves,
// three in a larger one, which keeps every warp full.  Trees of up to 2^13 leaves, whose time is one
// chain of compressions, run merkle_chain_kernel.  Upper layers
// run in CTAs that fuse up to 9 layers (512 inputs -> 1).  SHA-256 is pure integer work
// (funnel-shift rotates, three-input logic ops, adds).
#include <string.h>

#include <algorithm>
#include <mutex>

#include "host_sha256.h"
#include "internal.h"
#include "pdl.cuh"
#include "sha256.cuh"

using namespace bgpu;

namespace {

constexpr uint32_t kLeafFuse = 8;  // at most 2^8 leaves per CTA (Tuning::merkle_leaf_fuse)
constexpr uint32_t kNodeFuse = 9;  // at most 2^9 inputs per CTA (Tuning::merkle_node_fuse)
// From 2^17 inputs up a launch stops after three layers, where its 256-thread CTAs have a full warp
// left: the ALU pipe bounds it (SHA-256's rotates and three-input logic, 1024 of its 1376
// instructions), and the layers above would run the pipe for a warp with 16, 8, .. 1 lanes on.
// Measured on B200, all layers of a CTA -> three, in us: 2^24 leaves of one element 3147 -> 2458
// (13.7 G compressions/s), 2^22 819 -> 653, 2^20 237 -> 194, 2^20 of 16 elements 545 -> 471, 2^18 89
// -> 74, 2^17 64 -> 58; at 2^16 (47 -> 46) and below (2^15 33 -> 44) the added launches cost what the
// idle lanes do, or more.  Two or four layers are within 4% of three.  (Both sides with the last
// block's schedule as an argument; without that and with all layers 3278, 858, .., 579, 95.)
constexpr uint32_t kFullLog = 17;
constexpr uint32_t kFullLayers = 3;

__host__ __device__ __forceinline__ uint64_t layer_offset(uint32_t L, uint32_t k) {
  return (1ull << (L + 1)) - (1ull << (L + 1 - k));
}

__device__ __forceinline__ void store_digest(uint4* nodes, uint64_t i, const uint32_t d[8]) {
  nodes[2 * i] = make_uint4(d[0], d[1], d[2], d[3]);
  nodes[2 * i + 1] = make_uint4(d[4], d[5], d[6], d[7]);
}

__device__ __forceinline__ void load_digest(const uint4* nodes, uint64_t i, uint32_t d[8]) {
  uint4 a = nodes[2 * i], b = nodes[2 * i + 1];
  d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w;
  d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
}

// Hashes blockDim.x leaves per CTA and compresses `fused` layers above them in shared memory.
template <int N>
__global__ void __launch_bounds__(256) merkle_leaves_kernel(const uint4* __restrict__ elems,
                                                            uint32_t log_batch,
                                                            uint4* __restrict__ nodes, uint32_t L,
                                                            uint32_t fused, NodeIV iv,
                                                            PadSchedule pad) {
  pdl_wait();
  __shared__ uint32_t buf[2][256][9];  // padded rows avoid bank conflicts
  const uint32_t tid = threadIdx.x;
  const uint64_t leaf = (uint64_t)blockIdx.x * blockDim.x + tid;
  uint32_t d[8];
  sha256_elems<N>(elems + (leaf << log_batch), 1u << log_batch, pad, d);
  store_digest(nodes, leaf, d);
#pragma unroll
  for (int i = 0; i < 8; i++) buf[0][tid][i] = d[i];
  for (uint32_t lvl = 1; lvl <= fused; lvl++) {
    __syncthreads();
    const uint32_t n = blockDim.x >> lvl;
    if (tid < n) {
      const uint32_t src = (lvl - 1) & 1, dst = lvl & 1;
      uint32_t l[8], r[8], o[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        l[i] = buf[src][2 * tid][i];
        r[i] = buf[src][2 * tid + 1][i];
      }
      compress_node(iv, l, r, o);
#pragma unroll
      for (int i = 0; i < 8; i++) buf[dst][tid][i] = o[i];
      store_digest(nodes, layer_offset(L, lvl) + (uint64_t)blockIdx.x * n + tid, o);
    }
  }
}

// Compresses `fused` layers starting from layer in_level; a CTA has 2 blockDim.x inputs.
__global__ void __launch_bounds__(256) merkle_nodes_kernel(uint4* __restrict__ nodes, uint32_t L,
                                                           uint32_t in_level, uint32_t fused,
                                                           NodeIV iv) {
  pdl_wait();
  __shared__ uint32_t buf[2][256][9];
  const uint32_t tid = threadIdx.x;
  const uint64_t in_off = layer_offset(L, in_level);
  uint32_t l[8], r[8], o[8];
  {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + tid;
    load_digest(nodes, in_off + 2 * i, l);
    load_digest(nodes, in_off + 2 * i + 1, r);
    compress_node(iv, l, r, o);
    store_digest(nodes, layer_offset(L, in_level + 1) + i, o);
#pragma unroll
    for (int k = 0; k < 8; k++) buf[1][tid][k] = o[k];
  }
  for (uint32_t lvl = 2; lvl <= fused; lvl++) {
    __syncthreads();
    const uint32_t n = (blockDim.x * 2) >> lvl;
    if (tid < n) {
      const uint32_t src = (lvl - 1) & 1, dst = lvl & 1;
#pragma unroll
      for (int k = 0; k < 8; k++) {
        l[k] = buf[src][2 * tid][k];
        r[k] = buf[src][2 * tid + 1][k];
      }
      compress_node(iv, l, r, o);
#pragma unroll
      for (int k = 0; k < 8; k++) buf[dst][tid][k] = o[k];
      store_digest(nodes, layer_offset(L, in_level + lvl) + (uint64_t)blockIdx.x * n + tid, o);
    }
  }
}

// The last block of a message of n_elems elements, n_elems a multiple of 4.
PadSchedule pad_schedule(uint32_t n_elems) {
  PadSchedule p = {{0x80000000u}};
  p.w[15] = n_elems * 128u;
  auto rotr = [](uint32_t x, int n) { return (x >> n) | (x << (32 - n)); };
  for (int t = 16; t < 64; t++)
    p.w[t] = p.w[t - 16] + (rotr(p.w[t - 15], 7) ^ rotr(p.w[t - 15], 18) ^ (p.w[t - 15] >> 3)) +
             p.w[t - 7] + (rotr(p.w[t - 2], 17) ^ rotr(p.w[t - 2], 19) ^ (p.w[t - 2] >> 10));
  return p;
}

// ---- small trees
//
// A tree of few leaves is a chain: a leaf's blocks one after the other, then the layers.  One warp
// alone takes 2.1 k cycles a compression (1024 instructions of the half-rate ALU pipe, 8 of 18 a
// round for the message schedule), and two warps on one scheduler twice that.  Here a CTA has 32
// nodes, one to a lane, and only warp 0, alone on its scheduler, runs their rounds; warps 1, 2 and
// 3 prepare the schedules, block b on warp 1 + b mod 3, 16 words at a time through shared memory.
// A layer's schedule starts from the digests that warp 0 leaves in shared memory, while warp 0 runs
// the first 16 rounds from the same words.
//
// Measured on B200 against a thread per leaf and 256 leaves per CTA, in us with the launches: 2^8
// leaves of 64 elements 62 -> 29, 2^10 of 16 37 -> 20, 2^12 of 16 40 -> 24, 2^13 of 16 42 -> 28; at
// 2^14 they meet, where several of these CTAs share an SM and their first warps its scheduler, and
// above it loses (2^15 of one element 33 -> 47).  A compression of the chain takes 1.0 us.
constexpr uint32_t kChainMaxLog = 13;
constexpr uint32_t kChainLog = 5;  // a CTA's nodes
constexpr uint32_t kChainThreads = 128;
struct ChainShared {
  uint4 kw[3][16][32];  // K[t] + W[t] of block b mod 3, four words to a lane's element
  uint4 digests[2][32][2];
};
// Named barriers of warp 0 and a buffer's warp: words 16 c .. written (c < 4; c = 0 of a layer: its
// digests written, by warp 0), all words read (c = 4).
__device__ __forceinline__ uint32_t chain_bar(uint32_t buffer, uint32_t c) {
  return 1 + 5 * buffer + c;
}
__device__ __forceinline__ void chain_arrive(uint32_t id) {
  asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
}
__device__ __forceinline__ void chain_wait(uint32_t id) {
  asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}

// The words of lane's node of a layer above: the digests of nodes 2 lane and 2 lane + 1 below (lanes
// past the layer's end take others').
__device__ __forceinline__ void chain_children(const uint4 (&d)[32][2], uint32_t (&w)[16]) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint4 v = d[(2 * lane + i / 2) & 31][i & 1];
    w[4 * i + 0] = bswap32(v.x);
    w[4 * i + 1] = bswap32(v.y);
    w[4 * i + 2] = bswap32(v.z);
    w[4 * i + 3] = bswap32(v.w);
  }
}

// NODES = false: hashes 2^log_n leaves per CTA (log_n <= 5) and compresses the log_n layers above
// them.  NODES = true: compresses the log_n + 1 layers above layer in_level, 2^(log_n + 1) of its
// nodes per CTA.
template <bool NODES>
__global__ void __launch_bounds__(kChainThreads)
    merkle_chain_kernel(const uint4* __restrict__ elems, uint32_t log_batch,
                        uint4* __restrict__ nodes, uint32_t L, uint32_t in_level, uint32_t log_n,
                        NodeIV iv) {
  pdl_wait();
  pdl_trigger();
  __shared__ ChainShared sh;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x / 32, n = 1u << log_n;
  const uint32_t n_elems = 1u << log_batch;
  const uint32_t n_blocks = NODES ? 1 : n_elems / 4 + 1, total = n_blocks + log_n;
  const uint64_t first = (uint64_t)blockIdx.x << log_n;  // of this CTA's nodes of the lowest layer
  const uint64_t mine = first + (lane & (n - 1));
  if (warp) {
    for (uint32_t b = warp - 1; b < total; b += 3) {
      const uint32_t buf = warp - 1;
      // warp 0 is through with the buffer's last block, and so with that one's barriers
      if (b >= 3) chain_wait(chain_bar(buf, 4));
      uint32_t w[16];
      if (b >= n_blocks) {
        chain_wait(chain_bar(buf, 0));
        chain_children(sh.digests[(b - n_blocks) & 1], w);
      } else if (NODES) {
        const uint4* src = nodes + 2 * (layer_offset(L, in_level) + 2 * mine);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const uint4 v = src[i];
          w[4 * i + 0] = bswap32(v.x);
          w[4 * i + 1] = bswap32(v.y);
          w[4 * i + 2] = bswap32(v.z);
          w[4 * i + 3] = bswap32(v.w);
        }
      } else {
        const uint4* src = elems + (mine << log_batch);
        const uint32_t end = b + 1 == n_blocks;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const uint32_t e = 4 * b + i;
          uint4 v = make_uint4(e == n_elems ? 0x80u : 0u, 0u, 0u, 0u);
          if (e < n_elems) v = __ldg(src + e);
          w[4 * i + 0] = bswap32(v.x);
          w[4 * i + 1] = bswap32(v.y);
          w[4 * i + 2] = bswap32(v.z);
          w[4 * i + 3] = bswap32(v.w);
        }
        if (end) w[15] = n_elems * 128u;
      }
#pragma unroll 1
      for (uint32_t c = 0; c < 4; c++) {
        if (c) {
#pragma unroll
          for (int t = 0; t < 16; t++) {
            const uint32_t w15 = w[(t + 1) & 15], w2 = w[(t + 14) & 15];
            const uint32_t s0 = rotr32(w15, 7) ^ rotr32(w15, 18) ^ (w15 >> 3);
            const uint32_t s1 = rotr32(w2, 17) ^ rotr32(w2, 19) ^ (w2 >> 10);
            w[t] = w[t] + s0 + w[(t + 9) & 15] + s1;
          }
        } else if (b >= n_blocks) {
          continue;  // warp 0 has these words
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
          sh.kw[buf][4 * c + i][lane] = make_uint4(
              w[4 * i] + kSha256K[16 * c + 4 * i], w[4 * i + 1] + kSha256K[16 * c + 4 * i + 1],
              w[4 * i + 2] + kSha256K[16 * c + 4 * i + 2],
              w[4 * i + 3] + kSha256K[16 * c + 4 * i + 3]);
        chain_arrive(chain_bar(buf, c));
      }
    }
    return;
  }
  uint32_t s[8], buf = 0;
  if (NODES) {
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = iv.w[i];
  } else {
    sha256_init(s);
  }
  for (uint32_t b = 0; b < total; b++, buf = buf == 2 ? 0 : buf + 1) {
    const bool layer = b >= n_blocks;
    uint4 x[4];
    auto load = [&](uint32_t c) {
      chain_wait(chain_bar(buf, c));
#pragma unroll
      for (int i = 0; i < 4; i++) x[i] = sh.kw[buf][4 * c + i][lane];
    };
    if (layer) {
      uint32_t w[16];
      chain_children(sh.digests[(b - n_blocks) & 1], w);
#pragma unroll
      for (int i = 0; i < 4; i++)
        x[i] = make_uint4(w[4 * i] + kSha256K[4 * i], w[4 * i + 1] + kSha256K[4 * i + 1],
                          w[4 * i + 2] + kSha256K[4 * i + 2], w[4 * i + 3] + kSha256K[4 * i + 3]);
#pragma unroll
      for (int i = 0; i < 8; i++) s[i] = iv.w[i];
    } else {
      load(0);
    }
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = s[i];
    // unrolled, which lets the words' reads in among the rounds before: 1957 cycles a block, a loop of
    // four steps 2294, of two with the next step's words read ahead 2894
#pragma unroll
    for (uint32_t c = 0; c < 4; c++) {
      if (c) load(c);
      sha256_rounds16(v, reinterpret_cast<const uint32_t*>(x));
    }
    if (b + 3 < total) chain_arrive(chain_bar(buf, 4));
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] += v[i];
    if (b + 1 < n_blocks) continue;
    uint32_t o[8];
#pragma unroll
    for (int i = 0; i < 8; i++) o[i] = NODES || layer ? s[i] : bswap32(s[i]);
    const uint32_t up = b + 1 - n_blocks;
    if (up < log_n) {
      sh.digests[up & 1][lane][0] = make_uint4(o[0], o[1], o[2], o[3]);
      sh.digests[up & 1][lane][1] = make_uint4(o[4], o[5], o[6], o[7]);
      __syncwarp();
      chain_arrive(chain_bar(buf == 2 ? 0 : buf + 1, 0));
    }
    if (lane < n >> up)
      store_digest(nodes, layer_offset(L, in_level + up + (NODES ? 1 : 0)) + (first >> up) + lane,
                   o);
    __syncwarp();
  }
}

}  // namespace

namespace bgpu {

// Sha256Compression::default (hash/compress.rs:37-44): the digest bytes of
// "BINIUS SHA-256 COMPRESS" reinterpreted as native little-endian u32 words.
NodeIV node_iv() {
  static NodeIV iv;
  static std::once_flag once;
  std::call_once(once, [] {
    const char* tag = "BINIUS SHA-256 COMPRESS";
    uint8_t d[32];
    HostSha256::oneshot(reinterpret_cast<const uint8_t*>(tag), strlen(tag), d);
    for (int i = 0; i < 8; i++)
      iv.w[i] = (uint32_t)d[4 * i] | ((uint32_t)d[4 * i + 1] << 8) |
                ((uint32_t)d[4 * i + 2] << 16) | ((uint32_t)d[4 * i + 3] << 24);
  });
  return iv;
}

bool merkle_is_tuned(uint32_t log_leaves) { return log_leaves > kChainMaxLog; }

int merkle_commit(const void* d_elems, uint32_t log_leaves, uint32_t log_batch, void* d_nodes,
                  cudaStream_t stream) {
  BGPU_ARG(d_elems != nullptr && d_nodes != nullptr, "elems / nodes is NULL");
  BGPU_ARG(log_leaves <= 34, "too many leaves");
  BGPU_ARG(log_batch <= 20, "leaf too large");
  const uint32_t L = log_leaves;
  const NodeIV iv = node_iv();
  uint4* nodes = static_cast<uint4*>(d_nodes);
  if (L <= kChainMaxLog) {
    uint32_t level = std::min(L, kChainLog);
    auto launch = [&](auto kern, uint32_t grid_log, uint32_t in_level, uint32_t log_n) {
      cudaError_t e = launch_pdl(kern, 1u << grid_log, kChainThreads, 0, stream,
                                 static_cast<const uint4*>(d_elems), log_batch, nodes, L, in_level,
                                 log_n, iv);
      if (e != cudaSuccess) return cuda_error(e, "merkle_chain_kernel");
      count_launch();
      return (int)BINIUS_OK;
    };
    if (int rc = launch(merkle_chain_kernel<false>, L - level, 0, level)) return rc;
    while (level < L) {
      const uint32_t f = std::min(L - level, kChainLog + 1);
      if (int rc = launch(merkle_chain_kernel<true>, L - level - f, level, f - 1)) return rc;
      level += f;
    }
    return clear_error();
  }
  const uint32_t leaf_fuse = std::max(5u, std::min(kLeafFuse, tuning().merkle_leaf_fuse));
  const uint32_t node_fuse = std::max(5u, std::min(kNodeFuse, tuning().merkle_node_fuse));
  const uint32_t log_cta = std::min(L, leaf_fuse);
  const uint64_t grid = 1ull << (L - log_cta);
  BGPU_ARG(grid <= 0x7fffffffull, "too many leaves");
  auto layers = [](uint32_t log_inputs, uint32_t cta_layers) {
    return log_inputs >= kFullLog ? std::min(cta_layers, kFullLayers) : cta_layers;
  };
  const auto* elems = static_cast<const uint4*>(d_elems);
  uint32_t level = layers(L, log_cta);
  // the last block's schedule as an argument pays for large trees only: a small one's time is the
  // latency of a few warps, to which the reads of the argument add (1 us a launch)
  const bool large = L >= kFullLog;
  const PadSchedule pad = large ? pad_schedule(1u << log_batch) : PadSchedule{};
  auto kern = !large           ? merkle_leaves_kernel<0>
              : log_batch == 0 ? merkle_leaves_kernel<1>
              : log_batch == 1 ? merkle_leaves_kernel<2>
                               : merkle_leaves_kernel<4>;
  launch_pdl(kern, (unsigned)grid, 1u << log_cta, 0, stream, elems, log_batch, nodes, L, level, iv,
             pad);
  BGPU_LAUNCH_CHECK("merkle_leaves_kernel");
  count_launch();
  while (level < L) {
    const uint32_t f = std::min(L - level, node_fuse);
    const uint64_t g = 1ull << (L - level - f);
    const uint32_t fused = layers(L - level, f);
    launch_pdl(merkle_nodes_kernel, (unsigned)g, 1u << (f - 1), 0, stream, nodes, L, level, fused,
               iv);
    BGPU_LAUNCH_CHECK("merkle_nodes_kernel");
    count_launch();
    level += fused;
  }
  return clear_error();
}

}  // namespace bgpu

extern "C" {

int binius_merkle_commit(const void* d_elems, uint32_t log_leaves, uint32_t log_batch,
                         void* d_nodes, void* stream) {
  return bgpu::merkle_commit(d_elems, log_leaves, log_batch, d_nodes, as_stream(stream));
}

int binius_merkle_branch(const void* d_nodes, uint32_t log_leaves, uint64_t index,
                         uint32_t layer_depth, void* h_branch, void* stream) {
  BGPU_ARG(d_nodes != nullptr && h_branch != nullptr, "nodes / branch is NULL");
  BGPU_ARG(log_leaves <= 40, "log_leaves too large");
  BGPU_ARG(index < (1ull << log_leaves) && layer_depth <= log_leaves, "index out of range");
  cudaStream_t s = as_stream(stream);
  const uint8_t* nodes = static_cast<const uint8_t*>(d_nodes);
  uint8_t* out = static_cast<uint8_t*>(h_branch);
  for (uint32_t j = 0; j < log_leaves - layer_depth; j++) {
    uint64_t node = layer_offset(log_leaves, j) | ((index >> j) ^ 1);
    BGPU_CUDA(cudaMemcpyAsync(out + 32 * j, nodes + 32 * node, 32, cudaMemcpyDeviceToHost, s));
  }
  BGPU_CUDA(stream_wait(s));
  return clear_error();
}

int binius_merkle_layer(const void* d_nodes, uint32_t log_leaves, uint32_t layer_depth,
                        void* h_out, void* stream) {
  BGPU_ARG(d_nodes != nullptr && h_out != nullptr, "nodes / out is NULL");
  BGPU_ARG(log_leaves <= 40, "log_leaves too large");
  BGPU_ARG(layer_depth <= log_leaves, "IncorrectLayerDepth");
  // BinaryMerkleTree::layer: the 2^depth digests that end 2^depth - 1 digests before the end
  const uint64_t total = (2ull << log_leaves) - 1;
  const uint64_t start = total + 1 - (2ull << layer_depth);
  if (int rc = read_sync(h_out, static_cast<const uint8_t*>(d_nodes) + 32 * start,
                         32ull << layer_depth, as_stream(stream)))
    return rc;
  return clear_error();
}

}  // extern "C"
