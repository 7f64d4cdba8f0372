// Blake2s Merkle layer: MerkleOps<Blake2sMerkleHasher>::commit_on_layer.
//
// Node i of a layer of log size L is
//   Blake2s-256( prev[2i] || prev[2i+1] || col_0[i] || ... || col_{k-1}[i] )
// with the children only when a previous (larger) layer exists and each
// column value as 4 little-endian bytes (crates/stwo/src/core/vcs/
// blake2_merkle.rs:18-39, cpu/blake2s.rs:13-26).
//
// One thread hashes one node: its message block is built directly in
// registers from coalesced column reads (consecutive threads read
// consecutive rows of a column) and compressed in place; the children are
// read as 4 x 16-byte vector loads. No byte-wise buffering.
#include "runtime.cuh"
#include "blake2s.cuh"
#include "merkle_tail.cuh"
#include "channel.cuh"
#include <cstdlib>
#include <cstring>
#include <vector>
#include <algorithm>

namespace gs {

__device__ __forceinline__ void store_hash(uint32_t* out, size_t i, const uint32_t h[8]) {
  uint4* o = reinterpret_cast<uint4*>(out + 8 * i);
  o[0] = make_uint4(h[0], h[1], h[2], h[3]);
  o[1] = make_uint4(h[4], h[5], h[6], h[7]);
}

// FMA: adds of the compression on the FMA pipe (blake2s_compress_f). TABLE:
// columns through the pointer table, else from a base and a stride, chosen at
// compile time: a choice per word keeps a block's 16 loads from being issued
// together (64 columns x 2^20 rows, not 16-byte aligned: 308 us, now 196; 100
// x 2^13 29.5 -> 15.0). Five blocks per SM: 48 registers, where the compiler
// takes 55 to 59 by itself (2^19 nodes of two children 25.0 -> 23.8 us; 21.8
// with its launch overlapped).
template <bool FMA, bool TABLE>
__global__ void __launch_bounds__(256, 5)
    merkle_layer_kernel(uint32_t log_size, const uint32_t* __restrict__ prev, const uint32_t* const* __restrict__ tab,
                        const uint32_t* __restrict__ base, size_t stride, uint32_t n_cols, uint32_t* __restrict__ out,
                        uint32_t one) {
  const uint32_t prev_words = prev ? 16u : 0u;  // (before the shift: a null stays null)
  after_previous(prev, tab, base);
  const size_t n = (size_t)1 << log_size;
  const uint32_t total_words = prev_words + n_cols;
  const uint32_t total_bytes = 4u * total_words;
  const uint32_t n_blocks = total_words == 0 ? 1u : (total_words + 15u) / 16u;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    uint32_t h[8];
    blake2s_init(h);
    uint32_t m[16];
    uint32_t blk = 0;
    uint32_t col = 0;
    if (prev_words) {
      const uint4* p = reinterpret_cast<const uint4*>(prev + 16 * i);
      uint4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2), d = __ldg(p + 3);
      m[0] = a.x; m[1] = a.y; m[2] = a.z; m[3] = a.w;
      m[4] = b.x; m[5] = b.y; m[6] = b.z; m[7] = b.w;
      m[8] = c.x; m[9] = c.y; m[10] = c.z; m[11] = c.w;
      m[12] = d.x; m[13] = d.y; m[14] = d.z; m[15] = d.w;
      blk = 1;
      uint32_t t = total_bytes < 64u ? total_bytes : 64u;
      if (FMA) blake2s_compress_f(h, m, t, n_blocks == 1, one);
      else blake2s_compress(h, m, t, n_blocks == 1);
    }
    for (; blk < n_blocks; blk++) {
#pragma unroll
      for (int j = 0; j < 16; j++) {
        uint32_t c = col + j;
        m[j] = c < n_cols ? __ldg((TABLE ? tab[c] : base + c * stride) + i) : 0u;
      }
      col += 16;
      uint32_t t = 64u * (blk + 1);
      if (t > total_bytes) t = total_bytes;
      if (FMA) blake2s_compress_f(h, m, t, blk + 1 == n_blocks, one);
      else blake2s_compress(h, m, t, blk + 1 == n_blocks);
    }
    store_hash(out, i, h);
  }
}

// The same layer for 16-byte aligned columns of at least 32 rows. Bound by the
// ALU pipe inside the compression, so what goes is everything around it: a
// warp owns 32 rows and stages each message block (16 columns x 32 rows, 2
// KiB) in shared memory with four 16-byte cp.async per lane, one block ahead
// of the compression; a message word is then one conflict-free shared load at
// a constant offset, without a pointer load, address arithmetic and bounds
// check per word, and the columns' latency runs beside the compression. Only
// the warp itself reads its buffer, so no block barrier is needed. Columns
// past the last are zero-filled by the copy.
// 64 columns x 2^20 rows: 206 -> 179 us (23.4 compressions per ns; the ALU pipe
// alone would take 144 us).
constexpr int COL_WARPS = 4;
template <bool PREV>
__global__ void __launch_bounds__(32 * COL_WARPS, 8)
    merkle_columns_kernel(uint32_t log_size, const uint32_t* __restrict__ prev,
                          Cols cols, uint32_t n_cols, uint32_t* __restrict__ out, uint32_t one) {
  after_previous(prev);
  __shared__ uint4 stage[COL_WARPS][2][16 * 8];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t n_tiles = 1u << (log_size - 5), n_warps = gridDim.x * COL_WARPS;
  const uint32_t n_blocks = (n_cols + 15u) / 16u, total_bytes = 4u * n_cols + (PREV ? 64u : 0u);
  auto issue = [&](uint32_t tile, uint32_t blk, uint32_t slot) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint32_t row = 4 * q + (lane >> 3), c = 16 * blk + row;  // this lane's column of the block
      const uint32_t* src = cols[c < n_cols ? c : 0u] + 32 * (size_t)tile + 4 * (lane & 7u);
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&stage[warp][slot][8 * row + (lane & 7u)]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(c < n_cols ? 16 : 0)
                   : "memory");
    }
  };
  uint32_t tile = blockIdx.x * COL_WARPS + warp, slot = 0;
  if (tile >= n_tiles) return;
  issue(tile, 0, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (; tile < n_tiles; tile += n_warps) {
    const size_t i = 32 * (size_t)tile + lane;
    uint32_t h[8], m[16];
    blake2s_init(h);
    if (PREV) {
      const uint4* p = reinterpret_cast<const uint4*>(prev + 16 * i);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint4 c = __ldg(p + q);
        m[4 * q] = c.x; m[4 * q + 1] = c.y; m[4 * q + 2] = c.z; m[4 * q + 3] = c.w;
      }
      blake2s_compress_f(h, m, 64u, false, one);
    }
    for (uint32_t blk = 0; blk < n_blocks; blk++) {
      const bool last = blk + 1 == n_blocks;
      const uint32_t next_tile = last ? tile + n_warps : tile;
      if (next_tile < n_tiles) issue(next_tile, last ? 0u : blk + 1, slot ^ 1u);
      asm volatile("cp.async.commit_group;" ::: "memory");  // possibly empty: keeps the count uniform
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();  // the other lanes' copies of this block have landed too
      const uint32_t* w = reinterpret_cast<const uint32_t*>(stage[warp][slot]) + lane;
#pragma unroll
      for (int j = 0; j < 16; j++) m[j] = w[32 * j];
      __syncwarp();  // every lane has read the slot before the next copy into it
      uint32_t t = (PREV ? 64u : 0u) + 64u * (blk + 1);
      if (t > total_bytes) t = total_bytes;
      blake2s_compress_f(h, m, t, last, one);
      slot ^= 1u;
    }
    store_hash(out, i, h);
  }
}

// Lifted Merkle leaves (MerkleOpsLifted::build_leaves, crates/stwo/src/
// prover/backend/cpu/merkle_lifted.rs:12-77): leaf i of 2^lift hashes every
// column's value at its lifted index ((i >> (lift - log + 1)) << 1) + (i & 1),
// columns in increasing size order (the caller sorts, stably). One leaf per
// thread; message blocks are filled straight from the column loads.
__global__ void __launch_bounds__(256) merkle_lifted_leaves_kernel(uint32_t lift, const uint32_t* const* __restrict__ cols,
                                                                   const uint8_t* __restrict__ shifts, uint32_t n_cols,
                                                                   uint32_t* __restrict__ out, uint32_t one) {
  const size_t n = (size_t)1 << lift;
  const uint32_t total_bytes = 4u * n_cols;
  const uint32_t n_blocks = (n_cols + 15u) / 16u;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    uint32_t h[8], m[16];
    blake2s_init(h);
    uint32_t col = 0;
    for (uint32_t blk = 0; blk < n_blocks; blk++) {
#pragma unroll
      for (int j = 0; j < 16; j++) {
        uint32_t c = col + j;
        uint32_t v = 0;
        if (c < n_cols) {
          const uint32_t s = shifts[c];  // lift - log
          const size_t idx = ((i >> (s + 1)) << 1) + (i & 1);
          v = __ldg(cols[c] + idx);
        }
        m[j] = v;
      }
      col += 16;
      uint32_t t = 64u * (blk + 1);
      if (t > total_bytes) t = total_bytes;
      blake2s_compress_f(h, m, t, blk + 1 == n_blocks, one);
    }
    store_hash(out, i, h);
  }
}

int lifted_leaves(cudaStream_t st, uint32_t lift, const uint32_t* const* d_cols, const uint8_t* d_shifts,
                  uint32_t n_cols, uint32_t* d_out) {
  GS_REQUIRE(lift <= 30 && n_cols >= 1, "bad lifted leaf layer");
  GS_REQUIRE(((uintptr_t)d_out & 15) == 0, "hash buffers must be 16-byte aligned");
  size_t n = (size_t)1 << lift;
  size_t blocks = (n + 255) / 256;
  size_t cap = (size_t)num_sms() * 8;
  if (blocks > cap) blocks = cap;
  merkle_lifted_leaves_kernel<<<(unsigned)blocks, 256, 0, st>>>(lift, d_cols, d_shifts, n_cols, d_out, 1u);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}

int commit_on_layer(cudaStream_t st, uint32_t log_size, const uint32_t* d_prev, Cols cols, uint32_t n_cols, uint32_t* d_out, bool cols_aligned) {
  GS_REQUIRE(log_size <= 30, "layer log size out of range");
  GS_REQUIRE(d_out != nullptr, "null output");
  GS_REQUIRE(n_cols == 0 || cols.given(), "null column table");
  GS_REQUIRE(((uintptr_t)d_out & 15) == 0 && ((uintptr_t)d_prev & 15) == 0, "hash buffers must be 16-byte aligned");
  size_t n = (size_t)1 << log_size;
  int threads = 256;
  size_t blocks = (n + threads - 1) / threads;
  size_t cap = (size_t)num_sms() * 8;
  if (blocks > cap) blocks = cap;
  static const bool alu_only = [] {
    const char* e = getenv("GS_BLAKE_ALU");
    return e && e[0] == '1';
  }();
  // With children and at most 24 columns, large layers stay with a thread per
  // node: the staged kernel's warps wait for their children once per tile (one
  // column injected at 2^22 nodes 376 us staged, 352 not; at 2^19 48.3 and
  // 43.9; at 2^17 12.8 and 16.8; 32 columns at 2^20 142 and 144).
  const bool staged = cols_aligned && n_cols > 0 && log_size >= 5 && !(d_prev && n_cols <= 24 && log_size >= 18);
  if (staged && !alu_only) {
    const size_t tiles = n / (32 * COL_WARPS) ? n / (32 * COL_WARPS) : 1;
    const size_t resident = (size_t)num_sms() * 8;  // one wave; a warp walks its tiles, copies crossing from one to the next
    const unsigned grid = (unsigned)(tiles < resident ? tiles : resident);
    if (d_prev)
      launch_after(merkle_columns_kernel<true>, grid, 32 * COL_WARPS, 0, st, log_size, d_prev, cols, n_cols, d_out, 1u);
    else
      launch_after(merkle_columns_kernel<false>, grid, 32 * COL_WARPS, 0, st, log_size, d_prev, cols, n_cols, d_out, 1u);
  } else {
    const auto kernel = alu_only ? (cols.tab ? merkle_layer_kernel<false, true> : merkle_layer_kernel<false, false>)
                                 : (cols.tab ? merkle_layer_kernel<true, true> : merkle_layer_kernel<true, false>);
    launch_after(kernel, (unsigned)blocks, threads, 0, st, log_size, d_prev, cols.tab, cols.base, cols.stride, n_cols,
                 d_out, 1u);
  }
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}

// Node-only layers of a small tree in one launch of one 8-CTA thread-block
// cluster: starting from the layer of log size `top` (<= MERKLE_TAIL_LOG,
// already in memory), every layer down to the root, node = Blake2s(left ||
// right). Each CTA first computes its own eighth of the tree (layers top-1
// down to 3) with block barriers only, passing each level to the next through
// shared memory (and writing it to its global layer); after one cluster
// barrier, CTA 0 computes the last 3 layers from the 8 subtree roots. Below
// 2^11 nodes a per-layer launch is latency-bound; 8 SMs give the first levels
// enough throughput.
struct LayerPtrs { uint32_t* p[12]; };

// With `state`, the channel step (mix_root + draw_secure_felt) on the new
// root follows in the same launch (FRI layers).
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(1024) merkle_tail_kernel(uint32_t top, LayerPtrs layers,
                                                                                    uint32_t* state, uint32_t* root_copy,
                                                                                    uint32_t* felt, uint32_t one) {
  __shared__ uint4 buf[2][256];
  cg::cluster_group cluster = cg::this_cluster();
  cluster_tree_levels(top, layers.p, false, buf, cluster, one);
  __shared__ ChannelWords ch;
  __shared__ uint32_t quad_tab[40];
  if (state && cluster.block_rank() == 0 && threadIdx.x < 32) {
    const uint32_t j = threadIdx.x & 3u;
    blake2s_quad_table(quad_tab);
    channel_begin(ch, state);
    uint32_t h0 = layers.p[0][j], h1 = layers.p[0][4 + j];
    if (threadIdx.x < 4) {
      if (root_copy) {
        root_copy[j] = h0;
        root_copy[4 + j] = h1;
      }
      channel_root(ch, j, h0, h1);
    }
    __syncwarp();
    blake2s_quad(quad_tab, ch.mix, CHANNEL_MIX_BYTES, h0, h1);
    if (threadIdx.x < 4) channel_mixed(ch, j, h0, h1, state);
    __syncwarp();
    uint32_t draws = 0;
    do blake2s_quad(quad_tab, ch.draw, CHANNEL_DRAW_BYTES, h0, h1);
    while (!channel_drawn(ch, h0, h1, draws++, state, felt));
  }
}

// Every node layer of a tree in one launch. A unit is a 512-child subtree:
// a block of 128 threads hashes its 256 parents, then each level above
// through shared memory, down to the unit's root (9 levels), writing every
// level to its global layer. Stage 1 has one block per unit of the input
// layer. The block that finishes last among the units under one next-stage
// unit goes on to hash that unit from the global layer; it learns that it is
// last from a ticket (atomicInc after __threadfence, the counter wrapping
// back to 0 for the next launch). No block waits for another, so there is no
// spinning and nothing to bound. The block that writes the root runs the
// optional channel step. Critical path: one compression per level, four
// lanes to each where a level has at most 32 nodes (blake2s_quad): the trees of
// a 2^16 Wide-Fibonacci proof 24.6 -> 22.7 us each, a 2^20-leaf tree 94 -> 76
// us (its units are cheaper too: the upper levels of a unit leave warps idle).
struct TreePtrs { uint32_t* p[TREE_MAX_LOG + 1]; };
// Threads per 512-child unit: 128, each hashing two nodes of the unit's first
// level (452 us of tree kernels per Poseidon2 2^18 proof, against 464 us
// with 256 threads and 568 us with 64, all with a thread per node): half the
// warps wait at the barriers of the upper levels, and twice as many units fit
// on an SM.
constexpr int TREE_THREADS = 128;

template <int U, int TH>
__global__ void __launch_bounds__(TH, TH >= 256 ? 4 : 8)
    merkle_tree_kernel(uint32_t top, TreePtrs layers, uint32_t* counters, uint32_t* state, uint32_t* root_copy,
                       uint32_t* felt, uint32_t one) {
  const uint32_t zero = (uint32_t)after_previous();
  static_assert(TH >= 128, "four lanes for each of 32 nodes");
  __shared__ uint4 buf[2][1 << U];
  __shared__ ChannelWords ch;
  __shared__ uint32_t last, quad_tab[40];
  const uint32_t tid = threadIdx.x, j = tid & 3u;
  blake2s_quad_table(quad_tab);
  uint32_t in_log = top;
  uint32_t u = blockIdx.x + zero;
  uint32_t cnt_off = 0;
  for (;;) {
    const int out_log = in_log > U ? (int)in_log - U : 0;
    const bool channel = out_log == 0 && state;
    if (channel && tid < 32) channel_begin(ch, state);  // read by warp 0 after the root
    int cur = 0, rel = (int)in_log - 1 - out_log;  // the unit's 2^rel nodes of level out_log + rel
    bool first = true;                             // its children: the input layer
    for (; rel > 5; rel--) {
      const uint32_t n = 1u << rel;
#pragma unroll 1
      for (uint32_t i = tid; i < n; i += TH) {
        uint4 c[4];
        if (first) {
          // written before the launch, or by other blocks of this launch:
          // read at L2, not through the non-coherent path
          const uint4* src = reinterpret_cast<const uint4*>(layers.p[in_log]) + 4 * (((size_t)u << rel) + i);
#pragma unroll
          for (int q = 0; q < 4; q++) c[q] = __ldcg(src + q);
        } else {
#pragma unroll
          for (int q = 0; q < 4; q++) c[q] = buf[cur ^ 1][4 * i + q];
        }
        uint32_t h[8];
        hash_block16(c, 64, h, one);
        tail_store_hash(layers.p[out_log + rel], ((size_t)u << rel) + i, h);
        buf[cur][2 * i] = make_uint4(h[0], h[1], h[2], h[3]);
        buf[cur][2 * i + 1] = make_uint4(h[4], h[5], h[6], h[7]);
      }
      __syncthreads();
      cur ^= 1;
      first = false;
    }
    if (first) {  // a unit of at most 64 children
      const uint4* src = reinterpret_cast<const uint4*>(layers.p[in_log]) + 4 * ((size_t)u << rel);
      for (uint32_t i = tid; i < (4u << rel); i += TH) buf[cur ^ 1][i] = __ldcg(src + i);
      __syncthreads();
    }
    // Levels of at most 32 nodes, then the channel's mix (-1) and draw (-2):
    // latency alone counts, so four lanes take each compression; from 8 nodes
    // on warp 0 goes on alone, without block barriers. Quads past the level's
    // nodes hash words nobody uses.
    uint32_t draws = 0;
    while (rel >= (channel ? -2 : 0)) {
      if (rel <= 3 && tid >= 32) break;
      const uint32_t n = rel >= 0 ? 1u << rel : 1u, i = tid >> 2;
      if (tid < (4 * n > 32 ? 4 * n : 32)) {
        uint32_t h0, h1;
        blake2s_quad(quad_tab, rel >= 0 ? buf[cur ^ 1] + 4 * i : rel == -1 ? ch.mix : ch.draw,
                     rel == -2 ? CHANNEL_DRAW_BYTES : CHANNEL_MIX_BYTES, h0, h1);
        if (rel >= 0 && i < n) {
          uint32_t* to = layers.p[out_log + rel] + 8 * (((size_t)u << rel) + i);
          uint32_t* s = reinterpret_cast<uint32_t*>(buf[cur] + 2 * i);
          to[j] = s[j] = h0;
          to[4 + j] = s[4 + j] = h1;
        }
        if (rel == 0 && out_log == 0 && tid < 4) {
          if (root_copy) {
            root_copy[j] = h0;
            root_copy[4 + j] = h1;
          }
          if (channel) channel_root(ch, j, h0, h1);
        }
        if (rel == -1 && tid < 4) channel_mixed(ch, j, h0, h1, state);
        if (rel == -2 && !channel_drawn(ch, h0, h1, draws, state, felt)) {
          draws++;
          continue;
        }
      }
      if (rel > 3) __syncthreads();
      else __syncwarp();
      cur ^= 1;
      rel--;
    }
    if (out_log == 0) return;
    const uint32_t group_log = out_log > U ? (uint32_t)U : (uint32_t)out_log;
    const uint32_t next_u = u >> group_log;
    if (tid == 0) {
      __threadfence();  // this unit's root (written by lanes 0..3 of this warp) before the ticket
      const uint32_t ticket = atomicInc(counters + cnt_off + next_u, (1u << group_log) - 1u);
      last = ticket == (1u << group_log) - 1u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    cnt_off += 1u << (out_log - group_log);
    u = next_u;
    in_log = out_log;
  }
}

int commit_node_layers_ch(cudaStream_t st, uint32_t top_log, uint32_t* const* layers, uint32_t* d_counters,
                          uint32_t* d_state, uint32_t* d_root_copy, uint32_t* d_felt);

// ------------------------------------------------------------- work-list
// A tree of the work-list on the device: its columns and layers as offsets
// into one pointer pool.
struct MerkleWlItem {
  uint32_t col_off, n_cols, layer_off, log;
};

// Persistent grid: block b takes trees b, b + gridDim.x, ... of a list
// bucketed by decreasing size. Leaf i hashes the columns' values at row i
// (commit_on_layer without a previous layer: 16 column words per message
// block, the last block final); each node layer hashes pairs of the layer
// below from shared memory (two buffers: 2^log and 2^(log-1) hashes), every
// layer also stored to its global buffer.
__global__ void __launch_bounds__(256) merkle_worklist_kernel(const MerkleWlItem* __restrict__ items, uint32_t n_items,
                                                              void* const* __restrict__ pool, uint32_t max_log,
                                                              uint32_t one) {
  extern __shared__ uint4 sb[];
  uint4* const buf0 = sb;
  uint4* const buf1 = sb + 2 * (1u << max_log);
  for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {
    const MerkleWlItem w = items[it];
    const uint32_t* const* cols = reinterpret_cast<const uint32_t* const*>(pool + w.col_off);
    uint32_t* const* layers = reinterpret_cast<uint32_t* const*>(pool + w.layer_off);
    const uint32_t n = 1u << w.log;
    const uint32_t total_bytes = 4u * w.n_cols;
    const uint32_t n_blocks = (w.n_cols + 15u) / 16u;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      uint32_t h[8], m[16];
      blake2s_init(h);
      for (uint32_t blk = 0; blk < n_blocks; blk++) {
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const uint32_t c = 16 * blk + j;
          m[j] = c < w.n_cols ? __ldg(cols[c] + i) : 0u;
        }
        uint32_t t = 64u * (blk + 1);
        if (t > total_bytes) t = total_bytes;
        blake2s_compress_f(h, m, t, blk + 1 == n_blocks, one);
      }
      store_hash(layers[w.log], i, h);
      buf0[2 * i] = make_uint4(h[0], h[1], h[2], h[3]);
      buf0[2 * i + 1] = make_uint4(h[4], h[5], h[6], h[7]);
    }
    __syncthreads();
    bool in0 = true;  // the layer below sits in buf0
    for (int L = (int)w.log - 1; L >= 0; L--) {
      const uint4* in = in0 ? buf0 : buf1;
      uint4* out = in0 ? buf1 : buf0;
      for (uint32_t j = threadIdx.x; j < (1u << L); j += blockDim.x) {
        uint4 c[4];
#pragma unroll
        for (int q = 0; q < 4; q++) c[q] = in[4 * j + q];
        uint32_t h[8];
        hash_block16(c, 64, h, one);
        store_hash(layers[L], j, h);
        out[2 * j] = make_uint4(h[0], h[1], h[2], h[3]);
        out[2 * j + 1] = make_uint4(h[4], h[5], h[6], h[7]);
      }
      __syncthreads();
      in0 = !in0;
    }
    __syncthreads();  // the next tree reuses the buffers
  }
}

int merkle_worklist(Context& ctx, const MerkleItem* items, uint32_t n_items) {
  if (n_items == 0) return OK;
  GS_REQUIRE(items != nullptr, "null tree list");
  cudaStream_t st = ctx.stream;
  uint32_t count[MERKLE_WL_MAX_LOG + 1] = {0};
  for (uint32_t k = 0; k < n_items; k++) {
    const MerkleItem& x = items[k];
    GS_REQUIRE(x.cols && x.layers && x.n_cols >= 1, "a work-list tree needs columns and layers");
    GS_REQUIRE(x.log <= 30, "tree log size out of range");
    for (uint32_t c = 0; c < x.n_cols; c++) GS_REQUIRE(x.cols[c] != nullptr, "null column");
    for (uint32_t L = 0; L <= x.log; L++)
      GS_REQUIRE(x.layers[L] && ((uintptr_t)x.layers[L] & 15) == 0, "layer buffers must be 16-byte aligned");
    if (x.log <= MERKLE_WL_MAX_LOG) count[x.log]++;
  }
  // larger trees: the per-tree path
  for (uint32_t k = 0; k < n_items; k++) {
    const MerkleItem& x = items[k];
    if (x.log <= MERKLE_WL_MAX_LOG) continue;
    Cols cols;
    GS_TRY(ctx.columns(x.cols, x.n_cols, &cols));
    bool aligned = true;
    for (uint32_t c = 0; c < x.n_cols; c++) aligned = aligned && ((uintptr_t)x.cols[c] & 15) == 0;
    GS_TRY(commit_on_layer(st, x.log, nullptr, cols, x.n_cols, x.layers[x.log], aligned));
    GS_TRY(commit_node_layers(st, x.log, x.layers, ctx.tree_counters));
  }
  uint32_t first[MERKLE_WL_MAX_LOG + 1] = {0}, total = 0, max_log = 0;
  for (int lg = (int)MERKLE_WL_MAX_LOG; lg >= 0; lg--) {
    first[lg] = total;
    total += count[lg];
    if (count[lg] && max_log == 0) max_log = (uint32_t)lg;
  }
  if (total == 0) return OK;
  // one upload: the items, then the pointer pool (columns and layers)
  std::vector<MerkleWlItem> wl(total);
  std::vector<void*> pool;  // column pointers are only read
  for (uint32_t k = 0; k < n_items; k++) {
    const MerkleItem& x = items[k];
    if (x.log > MERKLE_WL_MAX_LOG) continue;
    MerkleWlItem w{(uint32_t)pool.size(), x.n_cols, 0, x.log};
    for (uint32_t c = 0; c < x.n_cols; c++) pool.push_back(const_cast<uint32_t*>(x.cols[c]));
    w.layer_off = (uint32_t)pool.size();
    for (uint32_t L = 0; L <= x.log; L++) pool.push_back(x.layers[L]);
    wl[first[x.log]++] = w;
  }
  const size_t o_pool = (wl.size() * sizeof(MerkleWlItem) + 15) & ~(size_t)15;
  const size_t bytes = o_pool + pool.size() * sizeof(void*);
  std::vector<uint8_t> up(bytes);
  memcpy(up.data(), wl.data(), wl.size() * sizeof(MerkleWlItem));
  memcpy(up.data() + o_pool, pool.data(), pool.size() * sizeof(void*));
  const void* d = nullptr;
  void* owned = nullptr;
  if (bytes <= ctx.ring_cap / 2) {
    GS_TRY(ctx.stage_bytes(up.data(), bytes, &d));
  } else {
    GS_TRY(ctx.alloc_async(bytes, &owned));
    GS_CUDA_TRY(cudaMemcpyAsync(owned, up.data(), bytes, cudaMemcpyHostToDevice, st));
    d = owned;
  }
  const size_t smem = (size_t)3 * 16 << max_log;  // 2^max_log + 2^(max_log - 1) hashes, reserved as 3 * 2^max_log uint4
  static OncePerDevice limit;
  GS_CUDA_TRY(allow_smem(limit, merkle_worklist_kernel, (size_t)3 * 16 << MERKLE_WL_MAX_LOG));
  const uint32_t per_sm = (uint32_t)std::min<size_t>(8, ((size_t)200 << 10) / smem);
  const uint32_t grid = (uint32_t)std::min<size_t>(wl.size(), (size_t)num_sms() * (per_sm ? per_sm : 1));
  merkle_worklist_kernel<<<grid, 256, smem, st>>>((const MerkleWlItem*)d, (uint32_t)wl.size(),
                                                  (void* const*)((const uint8_t*)d + o_pool), max_log, 1u);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  if (owned) GS_CUDA_TRY(cudaFreeAsync(owned, st));  // stream-ordered: after the kernel
  return OK;
}

int commit_node_layers(cudaStream_t st, uint32_t top_log, uint32_t* const* layers, uint32_t* d_counters) {
  return commit_node_layers_ch(st, top_log, layers, d_counters, nullptr, nullptr, nullptr);
}

static bool merkle_legacy() {
  static const bool legacy = [] {
    const char* e = getenv("GS_MERKLE_LEGACY");
    return e && e[0] == '1';
  }();
  return legacy;
}

int commit_node_layers_to(cudaStream_t st, uint32_t top_log, uint32_t* const* layers, uint32_t* d_counters,
                          uint32_t* root_out) {
  GS_REQUIRE(root_out != nullptr, "null root output");
  if (top_log == 0 || merkle_legacy()) {  // no tree kernel writes the root
    GS_TRY(commit_node_layers(st, top_log, layers, d_counters));
    GS_CUDA_TRY(cudaMemcpyAsync(root_out, layers[0], 32, cudaMemcpyDefault, st));
    return OK;
  }
  return commit_node_layers_ch(st, top_log, layers, d_counters, nullptr, root_out, nullptr);
}

// A tree of top_log <= TREE_MAX_LOG uses at most 2^(27 - 2U) + 2^(27 - 3U) + 1
// ticket counters for units of 2^U children (checked against TREE_COUNTERS).
int commit_node_layers_ch(cudaStream_t st, uint32_t top_log, uint32_t* const* layers, uint32_t* d_counters,
                          uint32_t* d_state, uint32_t* d_root_copy, uint32_t* d_felt) {
  GS_REQUIRE(top_log <= 30, "layer log size out of range");
  const bool legacy = merkle_legacy();
  if (!legacy) {
    uint32_t top = top_log;
    while (top > TREE_MAX_LOG) {  // layers above 2^27 nodes: one launch each
      GS_TRY(commit_on_layer(st, top - 1, layers[top], Cols(), 0, layers[top - 1]));
      top--;
    }
    if (top == 0) {
      GS_REQUIRE(d_state == nullptr, "channel step needs a tree of at least two leaves");
      return OK;
    }
    GS_REQUIRE(d_counters != nullptr, "tree kernel needs its counters");
    TreePtrs tp{};
    for (uint32_t k = 0; k <= top; k++) {
      GS_REQUIRE(((uintptr_t)layers[k] & 15) == 0, "hash buffers must be 16-byte aligned");
      tp.p[k] = layers[k];
    }
    // units of 2^9 children (timed with 256 threads): 2^8 (440 -> 464 us of tree
    // kernels per Poseidon2 2^18 proof), 2^7 (854 us) and 2^10 (449 us) were
    // slower
    constexpr int unit = 9;
    {  // ticket counters the continuation stages use
      size_t need = 0;
      for (uint32_t in = top; in > (uint32_t)unit;) {
        const uint32_t out = in - unit, g = out > (uint32_t)unit ? (uint32_t)unit : out;
        need += (size_t)1 << (out - g);
        in = out;
      }
      GS_REQUIRE(need <= TREE_COUNTERS, "tree too large for the ticket counters");
    }
    const uint32_t blocks = top > (uint32_t)unit ? 1u << (top - unit) : 1u;
    launch_after(merkle_tree_kernel<unit, TREE_THREADS>, blocks, TREE_THREADS, 0, st, top, tp, d_counters, d_state,
                 d_root_copy, d_felt, 1u);
    note_launch();
    GS_CUDA_TRY(cudaGetLastError());
    return OK;
  }
  // Layers of 2^11 nodes and more: one full-GPU launch each; the rest in
  // one cluster launch.
  uint32_t top = top_log;
  while (top > MERKLE_TAIL_LOG) {
    GS_TRY(commit_on_layer(st, top - 1, layers[top], Cols(), 0, layers[top - 1]));
    top--;
  }
  int L = (int)top - 1;
  uint32_t tail_top = (uint32_t)(L + 1);
  if (tail_top == 0) {  // a single node: it is the root already
    GS_REQUIRE(d_state == nullptr, "channel step needs a tree of at least two leaves");
    return OK;
  }
  LayerPtrs lp{};
  for (uint32_t k = 0; k <= tail_top && k < 12; k++) {
    GS_REQUIRE(((uintptr_t)layers[k] & 15) == 0, "hash buffers must be 16-byte aligned");
    lp.p[k] = layers[k];
  }
  merkle_tail_kernel<<<8, 1024, 0, st>>>(tail_top, lp, d_state, d_root_copy, d_felt, 1u);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}

}  // namespace gs
