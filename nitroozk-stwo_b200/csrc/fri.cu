// FRI folds over QM31 columns stored as 4 coordinate planes.
//
// fold_line (crates/stwo/src/prover/backend/cpu/fri.rs:64-86):
//   for pair i of a line evaluation on half_odds(n) in bit-reversed order,
//   f0 = f(x) + f(-x), f1 = (f(x) - f(-x)) / x, out[i] = f0 + alpha f1,
//   with 1/x read from the itwiddle level of half_odds(n) (offset L - 2^n).
// fold_circle_into_line (cpu/fri.rs:88-113):
//   f0 = f(p) + f(-p), f1 = (f(p) - f(-p)) / p.y,
//   dst[i] = dst[i] alpha^2 + f0 + alpha f1,
//   with 1/p.y the circle-layer itwiddle of the domain (the same derivation
//   the interpolation's first layer uses).
//
// Fusion: when `leaf_out` is given, the thread that produced element i also
// hashes it as the Merkle leaf of the next FRI layer (Blake2s of the 4
// coordinates, one compression), so the folded layer is not read again for
// its leaf hashes.
#include "runtime.cuh"
#include "blake2s.cuh"
#include "channel.cuh"
#include "merkle_tail.cuh"

namespace gs {

__device__ __forceinline__ void leaf_hash4(uint32_t* leaf_out, size_t i, qm31 v, uint32_t one) {
  uint32_t h[8], m[16];
  blake2s_init(h);
  m[0] = v.x.a; m[1] = v.x.b; m[2] = v.y.a; m[3] = v.y.b;
  blake2s_compress_f<4>(h, m, 16, true, one);
  uint4* o = reinterpret_cast<uint4*>(leaf_out + 8 * i);
  o[0] = make_uint4(h[0], h[1], h[2], h[3]);
  o[1] = make_uint4(h[4], h[5], h[6], h[7]);
}

__device__ __forceinline__ void load_pair(CPlanes s, size_t i, qm31& a, qm31& b) {
  uint2 p0 = __ldg(reinterpret_cast<const uint2*>(s.p[0]) + i);
  uint2 p1 = __ldg(reinterpret_cast<const uint2*>(s.p[1]) + i);
  uint2 p2 = __ldg(reinterpret_cast<const uint2*>(s.p[2]) + i);
  uint2 p3 = __ldg(reinterpret_cast<const uint2*>(s.p[3]) + i);
  a = qm_make(p0.x, p1.x, p2.x, p3.x);
  b = qm_make(p0.y, p1.y, p2.y, p3.y);
}

// d_alpha (optional): the challenge in device memory (4 words, then alpha^2),
// written by the device channel; overrides `alpha`.
__global__ void fold_line_kernel(CPlanes src, uint32_t log_n, qm31 alpha, Planes dst, const uint32_t* __restrict__ itw,
                                 uint32_t tw_len, uint32_t* leaf_out, const uint32_t* __restrict__ d_alpha, uint32_t one) {
  after_previous(src, itw, d_alpha);
  const size_t half = (size_t)1 << (log_n - 1);
  if (d_alpha) alpha = qm_make(d_alpha[0], d_alpha[1], d_alpha[2], d_alpha[3]);
  const uint32_t* lvl = itw + (tw_len - (1u << log_n));
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < half; i += (size_t)gridDim.x * blockDim.x) {
    qm31 fx, fnx;
    load_pair(src, i, fx, fnx);
    uint32_t xinv = __ldg(lvl + i);
    qm31 f0 = qm_add(fx, fnx);
    qm31 f1 = qm_mul_m31(qm_sub(fx, fnx), xinv);
    qm31 r = qm_add(f0, qm_mul(alpha, f1));
    dst.p[0][i] = r.x.a; dst.p[1][i] = r.x.b; dst.p[2][i] = r.y.a; dst.p[3][i] = r.y.b;
    if (leaf_out) leaf_hash4(leaf_out, i, r, one);
  }
}

struct SmallInvY { uint32_t v[2]; };

__global__ void fold_circle_kernel(CPlanes src, uint32_t log_n, qm31 alpha, qm31 alpha_sq, Planes dst,
                                   const uint32_t* __restrict__ itw, uint32_t tw_len, SmallInvY small,
                                   uint32_t* leaf_out, const uint32_t* __restrict__ d_alpha, uint32_t one,
                                   uint32_t fresh) {
  after_previous(src, itw, d_alpha);
  const size_t half = (size_t)1 << (log_n - 1);
  if (d_alpha) {
    alpha = qm_make(d_alpha[0], d_alpha[1], d_alpha[2], d_alpha[3]);
    alpha_sq = qm_make(d_alpha[4], d_alpha[5], d_alpha[6], d_alpha[7]);
  }
  const uint32_t* t0 = log_n >= 3 ? itw + (tw_len - (1u << (log_n - 1))) : nullptr;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < half; i += (size_t)gridDim.x * blockDim.x) {
    qm31 fp, fnp;
    load_pair(src, i, fp, fnp);
    uint32_t yinv;
    if (t0) {
      uint32_t q = (uint32_t)(i >> 2), r = (uint32_t)(i & 3);
      uint32_t x = __ldg(t0 + 2 * q + (r < 2 ? 1u : 0u));
      yinv = (r == 1 || r == 2) ? neg(x) : x;
    } else {
      yinv = small.v[i];
    }
    qm31 f0 = qm_add(fp, fnp);
    qm31 f1 = qm_mul_m31(qm_sub(fp, fnp), yinv);
    qm31 fprime = qm_add(qm_mul(alpha, f1), f0);
    qm31 r = fprime;
    if (!fresh) {  // (a fresh dst counts as zero and is not read)
      qm31 d = qm_make(dst.p[0][i], dst.p[1][i], dst.p[2][i], dst.p[3][i]);
      r = qm_add(qm_mul(d, alpha_sq), fprime);
    }
    dst.p[0][i] = r.x.a; dst.p[1][i] = r.x.b; dst.p[2][i] = r.y.a; dst.p[3][i] = r.y.b;
    if (leaf_out) leaf_hash4(leaf_out, i, r, one);
  }
}

static unsigned grid_for(size_t n, int threads) {
  size_t b = (n + threads - 1) / threads;
  size_t cap = (size_t)num_sms() * 16;
  return (unsigned)(b < cap ? (b ? b : 1) : cap);
}

static int fold_line_launch(cudaStream_t st, CPlanes src, uint32_t log_n, qm31 alpha, Planes dst,
                            const uint32_t* d_itw, uint32_t tw_log, uint32_t* leaf_out, const uint32_t* d_alpha) {
  GS_REQUIRE(log_n >= 1 && log_n <= tw_log, "fold_line: line domain must fit the twiddle tree");
  size_t half = (size_t)1 << (log_n - 1);
  launch_after(fold_line_kernel, grid_for(half, 256), 256, 0, st, src, log_n, alpha, dst, d_itw,
               1u << tw_log, leaf_out, d_alpha, 1u);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}

static pt31 host_point(uint32_t k) {
  pt31 r = {1u, 0u}, cur = {2u, 1268011823u};
  for (int b = 0; b < 31; b++) {
    if ((k >> b) & 1u) r = pt_add(r, cur);
    cur = pt_add(cur, cur);
  }
  return r;
}

int fold_line_fused(cudaStream_t st, CPlanes src, uint32_t log_n, qm31 alpha, Planes dst, const uint32_t* d_itw,
                    uint32_t tw_log, uint32_t* leaf_out) {
  return fold_line_launch(st, src, log_n, alpha, dst, d_itw, tw_log, leaf_out, nullptr);
}
int fold_line_dev_alpha(cudaStream_t st, CPlanes src, uint32_t log_n, const uint32_t* d_alpha, Planes dst,
                        const uint32_t* d_itw, uint32_t tw_log, uint32_t* leaf_out) {
  return fold_line_launch(st, src, log_n, qm_zero(), dst, d_itw, tw_log, leaf_out, d_alpha);
}

static int fold_circle_launch(cudaStream_t st, CPlanes src, uint32_t log_n, qm31 alpha, Planes dst,
                              const uint32_t* d_itw, uint32_t tw_log, uint32_t* leaf_out, const uint32_t* d_alpha,
                              bool fresh = false) {
  GS_REQUIRE(log_n >= 1 && log_n <= tw_log + 1, "fold_circle_into_line: domain must fit the twiddle tree");
  SmallInvY small{{0, 0}};
  if (log_n < 3) {
    // CanonicCoset(n) half coset: initial index 2^(31-(n+1)), step 2^(31-(n-1)).
    uint32_t init = 1u << (31 - (log_n + 1)), step = log_n >= 2 ? 1u << (31 - (log_n - 1)) : 0u;
    for (uint32_t i = 0; i < (1u << (log_n - 1)); i++) {
      uint32_t j = (log_n - 1) ? ((i & 1) ? 1u : 0u) : 0u;  // bit-reverse over n-1 <= 1 bits
      pt31 p = host_point((init + j * step) & 0x7fffffffu);
      small.v[i] = inv(p.y);
    }
  }
  qm31 alpha_sq = qm_mul(alpha, alpha);
  size_t half = (size_t)1 << (log_n - 1);
  launch_after(fold_circle_kernel, grid_for(half, 256), 256, 0, st, src, log_n, alpha, alpha_sq, dst, d_itw,
               1u << tw_log, small, leaf_out, d_alpha, 1u, fresh ? 1u : 0u);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}
int fold_circle_into_line_fused(cudaStream_t st, CPlanes src, uint32_t log_n, qm31 alpha, Planes dst,
                                const uint32_t* d_itw, uint32_t tw_log, uint32_t* leaf_out) {
  return fold_circle_launch(st, src, log_n, alpha, dst, d_itw, tw_log, leaf_out, nullptr);
}
// The same into planes that hold nothing yet (dst counts as zero).
int fold_circle_fresh(cudaStream_t st, CPlanes src, uint32_t log_n, qm31 alpha, Planes dst, const uint32_t* d_itw,
                      uint32_t tw_log) {
  return fold_circle_launch(st, src, log_n, alpha, dst, d_itw, tw_log, nullptr, nullptr, true);
}
int fold_circle_fresh_dev_alpha(cudaStream_t st, CPlanes src, uint32_t log_n, const uint32_t* d_alpha, Planes dst,
                                const uint32_t* d_itw, uint32_t tw_log, uint32_t* leaf_out) {
  return fold_circle_launch(st, src, log_n, qm_zero(), dst, d_itw, tw_log, leaf_out, d_alpha, true);
}

// Fused tail of the FRI commit phase: every layer of log size <= 11 in one
// launch of one 1024-thread CTA. For layer k (log size log0 - k, leaves
// already hashed): its Merkle node levels (at most 1024 nodes each), the
// channel step on its root, then fold_line into layer k + 1 with that layer's
// leaf hashes — the steps the per-layer kernels run, with the data in shared
// memory and block barriers between them. The tail is a chain of about a
// hundred dependent steps, most of them one Blake2s compression long, so the
// latency of a compression bounds it: levels (and leaf layers) of at most 32
// hashes and the channel step take four lanes per compression (blake2s_quad),
// on warps 0..3 down to warp 0 alone; larger ones a thread each. The tail of a
// 2^16 or larger first layer: 144 -> 124 us, of a 2^11 one 112 -> 94 us. An
// 8-CTA cluster spent more on cluster barriers and L2 re-reads than it gained
// in width (164 against 132 us, a thread per hash in both).
// Shared memory (uint4): two hash buffers (2048: a layer's leaves, then its
// levels in turn), this layer's and the next one's values (1024 QM31 each) and
// 32 leaf messages.
constexpr uint32_t TAIL_CTA_SMEM = (2 * 2048 + 2 * 1024 + 32 * 4) * 16;
__device__ __forceinline__ void bar_sync_128() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
__global__ void __launch_bounds__(1024) fri_tail_cta_kernel(FriTail a, uint32_t* state,
                                                            const uint32_t* __restrict__ itw, uint32_t tw_len,
                                                            uint32_t one) {
  const uint32_t zero = (uint32_t)after_previous(itw);
  extern __shared__ uint4 tsm[];
  __shared__ ChannelWords ch;
  __shared__ uint32_t quad_tab[40];
  auto hashes = [&](int i) { return tsm + 2048 * i; };
  auto vals = [&](uint32_t i) { return tsm + 4096 + 1024 * i; };
  uint4* const msgs = tsm + 6144;
  const uint32_t tid = threadIdx.x + zero, j = tid & 3u;
  blake2s_quad_table(quad_tab);
  if (tid < 32) {
    channel_begin(ch, state);  // read by warp 0 after a root
    for (int q = 0; q < 4; q++) msgs[4 * tid + q] = make_uint4(0, 0, 0, 0);
  }
  for (uint32_t k = 0; k <= a.n; k++) {
    const uint32_t log = a.log0 - k;
    uint32_t* const* tree = a.tree[k];
    uint4 v;  // this thread's value of the layer
    if (k > 0 && tid < (1u << log)) {  // the fold of the layer before
      qm31 fx, fnx;
      if (k == 1) {  // layer 0's values come from the previous kernel
        uint32_t* const* sp = a.planes[0];
        fx = qm_make(__ldg(sp[0] + 2 * tid), __ldg(sp[1] + 2 * tid), __ldg(sp[2] + 2 * tid), __ldg(sp[3] + 2 * tid));
        fnx = qm_make(__ldg(sp[0] + 2 * tid + 1), __ldg(sp[1] + 2 * tid + 1), __ldg(sp[2] + 2 * tid + 1),
                      __ldg(sp[3] + 2 * tid + 1));
      } else {
        const uint4 p = vals((k - 1) & 1)[2 * tid], q = vals((k - 1) & 1)[2 * tid + 1];
        fx = qm_make(p.x, p.y, p.z, p.w);
        fnx = qm_make(q.x, q.y, q.z, q.w);
      }
      const qm31 alpha = qm_make(ch.felt.x, ch.felt.y, ch.felt.z, ch.felt.w);
      const uint32_t xinv = __ldg(itw + (tw_len - (2u << log)) + tid);
      const qm31 f0 = qm_add(fx, fnx);
      const qm31 f1 = qm_mul_m31(qm_sub(fx, fnx), xinv);
      const qm31 r = qm_add(f0, qm_mul(alpha, f1));
      uint32_t* const* dp = a.planes[k];
      dp[0][tid] = r.x.a; dp[1][tid] = r.x.b; dp[2][tid] = r.y.a; dp[3][tid] = r.y.b;
      v = make_uint4(r.x.a, r.x.b, r.y.a, r.y.b);
      vals(k & 1)[tid] = v;
      if (log <= 5) msgs[4 * tid] = v;
    }
    if (k == a.n) return;  // the last layer is not committed
    // s = log: the leaves (layer 0's were hashed by the previous kernel); s <
    // log: the 2^s nodes of level s, one thread each while there are more than 32
    int s = k == 0 ? (int)log - 1 : (int)log, cur = 0;
    for (; s > 5; s--) {
      if (tid < (1u << s)) {
        uint4 c[4];
        if (s == (int)log) {
          c[0] = v;
          c[1] = c[2] = c[3] = make_uint4(0, 0, 0, 0);
        } else if (s == (int)log - 1 && k == 0) {
          const uint4* src = reinterpret_cast<const uint4*>(tree[log]) + 4 * (size_t)tid;
#pragma unroll
          for (int q = 0; q < 4; q++) c[q] = __ldg(src + q);
        } else {
#pragma unroll
          for (int q = 0; q < 4; q++) c[q] = hashes(cur ^ 1)[4 * tid + q];
        }
        uint32_t h[8];
        hash_block16(c, s == (int)log ? 16u : 64u, h, one);
        tail_store_hash(tree[s], tid, h);
        hashes(cur)[2 * tid] = make_uint4(h[0], h[1], h[2], h[3]);
        hashes(cur)[2 * tid + 1] = make_uint4(h[4], h[5], h[6], h[7]);
      }
      __syncthreads();
      cur ^= 1;
    }
    if (tid < 128) {
      if (k == 0 && log <= 6) {  // a small first layer: its leaves
        const uint4* src = reinterpret_cast<const uint4*>(tree[log]);
        for (uint32_t i = tid; i < (2u << log); i += 128) hashes(cur ^ 1)[i] = __ldg(src + i);
      }
      bar_sync_128();  // the leaves or messages of the other warps
      uint32_t draws = 0;
      while (s >= -2) {
        if (s <= 3 && tid >= 32) break;
        const uint32_t n = s >= 0 ? 1u << s : 1u, i = tid >> 2;
        if (tid < (4 * n > 32 ? 4 * n : 32)) {
          const bool leaf = s == (int)log;
          uint32_t h0, h1;
          blake2s_quad(quad_tab, s >= 0 ? (leaf ? msgs : hashes(cur ^ 1)) + 4 * i : s == -1 ? ch.mix : ch.draw,
                       leaf ? 16u : s == -2 ? CHANNEL_DRAW_BYTES : 64u, h0, h1);
          if (s >= 0 && i < n) {
            uint32_t* to = tree[s] + 8 * (size_t)i;
            uint32_t* sh = reinterpret_cast<uint32_t*>(hashes(cur) + 2 * i);
            to[j] = sh[j] = h0;
            to[4 + j] = sh[4 + j] = h1;
          }
          if (s == 0 && tid < 4) {
            a.roots[8 * k + j] = h0;
            a.roots[8 * k + 4 + j] = h1;
            channel_root(ch, j, h0, h1);
          }
          if (s == -1 && tid < 4) channel_mixed(ch, j, h0, h1, state);
          if (s == -2 && !channel_drawn(ch, h0, h1, draws, state, a.felts + 8 * k)) {
            draws++;
            continue;
          }
        }
        if (s > 3) bar_sync_128();
        else __syncwarp();
        cur ^= 1;
        s--;
      }
    }
    __syncthreads();  // the challenge
  }
}

int fri_tail(cudaStream_t st, const FriTail& a, uint32_t* d_state, const uint32_t* d_itw, uint32_t tw_log) {
  GS_REQUIRE(a.n >= 1 && a.n <= FRI_TAIL_MAX && a.log0 <= FRI_TAIL_MAX - 1 && a.log0 >= a.n,
             "FRI tail: layer sizes out of range");
  GS_REQUIRE(a.log0 <= tw_log, "FRI tail: line domain must fit the twiddle tree");
  static OncePerDevice smem;
  GS_CUDA_TRY(allow_smem(smem, fri_tail_cta_kernel, TAIL_CTA_SMEM));
  launch_after(fri_tail_cta_kernel, 1, 1024, TAIL_CTA_SMEM, st, a, d_state, d_itw, 1u << tw_log, 1u);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}

}  // namespace gs
