// Batched circle FFT (interpolate / evaluate) over M31 columns.
//
// Semantics: crates/stwo/src/prover/backend/cpu/circle.rs:28-80 (interpolate)
// and :182-228 (evaluate). Layer i pairs index v with v + 2^i and uses the
// twiddle of group h = v >> (i + 1):
//   line layer i >= 1:  buf[L - 2^(n-i) + h]           (domain_line_twiddles_from_tree)
//   circle layer i = 0: from the first line slice T0,  h = 4q + r ->
//                       [T0[2q+1], -T0[2q+1], -T0[2q], T0[2q]][r]
// with buf = itwiddles for interpolation and twiddles for evaluation, L the
// twiddle buffer length. Interpolation runs layers 0..n-1 then scales by
// 1/2^n; evaluation runs layers n-1..0.
//
// Kernel design (radix-2^R in registers): a pass covers L consecutive layers
// on tiles of 2^t = 2^(c+L) elements. Each thread holds 2^R elements (R = 5:
// 32 registers) whose tile indices differ in an R-bit window and runs up to R
// layers on them with compile-time indexing; stages exchange data through
// shared memory with an XOR swizzle (bank = e[0:5] ^ e[5:10]) that keeps
// every access pattern bank-conflict free. The twiddles a thread needs for
// one layer are consecutive and aligned in the tree, so they arrive as a few
// 16-byte loads. A tile keeps its c lowest index bits contiguous in global
// memory (64-byte runs with c = 4) so strided passes read whole sectors.
// Columns of one size are batched in one launch (grid.y = column). The 1/2^n
// scale is fused into the final store of the interpolation.
//
// Low-degree extension (evaluate 2^m coefficients on a 2^n domain): the top
// n-m layers of the zero-padded forward FFT only copy (butterfly with a zero
// partner), so the first pass reads src[v mod 2^m] and only layers m-1..0
// are computed — no zero-extension pass.
#include "runtime.cuh"
#include <algorithm>
#include <vector>
#include <iterator>
#include <cstdlib>

namespace gs {

struct FftPass {
  uint32_t n;           // domain log size
  uint32_t lo, L;       // layers [lo, lo + L)
  uint32_t c;           // contiguous low index bits kept per tile (c <= lo)
  uint32_t t;           // tile log size = c + L
  uint32_t K;           // register stages
  uint32_t tile_shift;  // log2(tiles per block)
  uint32_t src_mask;    // read src[v & src_mask] (LDE replication)
  uint32_t tw_len;      // twiddle buffer length
  uint32_t scale;       // multiply by scale on the final store when has_scale
  uint32_t has_scale;
  uint32_t vec_ok;      // all column pointers 16-byte aligned: vector loads/stores allowed
};

__device__ __forceinline__ uint32_t circle_twiddle(const uint32_t* __restrict__ tw, uint32_t tw_len, uint32_t n,
                                                   uint32_t h) {
  uint32_t base = tw_len - (1u << (n - 1));
  uint32_t q = h >> 2, r = h & 3u;
  uint32_t x = __ldg(tw + base + 2 * q + (r < 2 ? 1u : 0u));
  return (r == 1 || r == 2) ? neg(x) : x;
}

// COUNT consecutive twiddles of layer i starting at group hth (aligned to COUNT).
template <int COUNT>
__device__ __forceinline__ void load_twiddles(uint32_t* w, const uint32_t* __restrict__ tw, uint32_t tw_len,
                                              uint32_t n, uint32_t i, uint32_t hth) {
  if (i >= 1) {
    const uint32_t* p = tw + (tw_len - (1u << (n - i)) + hth);
    if (COUNT >= 4) {
#pragma unroll
      for (int g = 0; g < COUNT / 4; g++) {
        uint4 v = __ldg(reinterpret_cast<const uint4*>(p) + g);
        w[4 * g] = v.x; w[4 * g + 1] = v.y; w[4 * g + 2] = v.z; w[4 * g + 3] = v.w;
      }
    } else if (COUNT == 2) {
      uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
      w[0] = v.x; w[1] = v.y;
    } else {
      w[0] = __ldg(p);
    }
  } else {
    if (COUNT >= 4) {
      const uint32_t* t0 = tw + (tw_len - (1u << (n - 1)));
#pragma unroll
      for (int g = 0; g < COUNT / 4; g++) {
        uint2 xy = __ldg(reinterpret_cast<const uint2*>(t0) + (hth >> 2) + g);
        w[4 * g] = xy.y; w[4 * g + 1] = neg(xy.y); w[4 * g + 2] = neg(xy.x); w[4 * g + 3] = xy.x;
      }
    } else {
#pragma unroll
      for (int g = 0; g < COUNT; g++) w[g] = circle_twiddle(tw, tw_len, n, hth + g);
    }
  }
}

template <bool INV>
__device__ __forceinline__ void bfly(uint32_t& a, uint32_t& b, uint32_t w) {
  if (INV) {
    uint32_t t0 = a;
    a = add(t0, b);
    b = mul(sub(t0, b), w);
  } else {
    uint32_t t0 = mul(b, w);
    b = sub(a, t0);
    a = add(a, t0);
  }
}

// Butterflies with one reduction less than three: on centred twiddles (s = 2w,
// less 2p where w > p/2: an even word in [2 - p, p - 1] as a signed one) the
// product of a signed b in [-p, p] comes out as t = b w (mod p) in [-p, p - 1]
// without any: b s + 2^31 - 2^62 has the high word b w / 2^31, rounded, less
// 2^30, and the low word half of which is the rest, plus 2^30.
__host__ __device__ __forceinline__ uint32_t centred2(uint32_t w) { return 2u * (w + (w >> 30)); }
__device__ __forceinline__ uint32_t mul_centred(uint32_t b, uint32_t s) {
  const int64_t p = (int64_t)(int32_t)b * (int32_t)s + ((1ll << 31) - (1ll << 62));
  return (uint32_t)((uint64_t)p >> 32) + ((uint32_t)p >> 1);
}
// Inverse, a and b canonical before and after: a - b needs no reduction.
__device__ __forceinline__ void bfly_inv(uint32_t& a, uint32_t& b, uint32_t s) {
  const uint32_t t = mul_centred(a - b, s);
  a = add(a, b);
  b = __viaddmin_u32(t, P, t);
}
// Forward: t goes to [-p, -1] and a to [0, p - 1], one step each, so that a + t
// is a signed word in [-p, p - 2] and a - t an unsigned one in [1, 2p - 1]. The
// next layer is told which of the two forms its operands have.
template <bool UNSIGNED>
__device__ __forceinline__ void bfly_fwd(uint32_t& a, uint32_t& b, uint32_t s) {
  uint32_t t = mul_centred(UNSIGNED ? b - P : b, s);
  t = __viaddmax_u32(t, 0u - P, t);
  const uint32_t r = __viaddmin_u32(a, UNSIGNED ? 0u - P : P, a);
  a = r + t;
  b = r - t;
}

// XOR swizzle over the block's shared-memory index (tile offset included, so
// blocks holding several small tiles stay conflict free as well).
__device__ __forceinline__ uint32_t swz(uint32_t e) { return e ^ ((e >> 5) & 31u); }

template <bool INV, int R>
__global__ void __launch_bounds__(256) fft_pass_kernel(Cols src_tab, MutCols dst_tab,
                                                       const uint32_t* __restrict__ tw, FftPass a) {
  extern __shared__ uint32_t sm[];
  constexpr int NQ = 1 << R;
  const uint32_t col = blockIdx.y;
  const uint32_t* __restrict__ src = src_tab[col];
  uint32_t* __restrict__ dst = dst_tab[col];
  const uint32_t tpt_log = a.t - R;
  const uint32_t ltid = threadIdx.x & ((1u << tpt_log) - 1u);
  const uint32_t sub_tile = threadIdx.x >> tpt_log;
  const uint32_t tile = (blockIdx.x << a.tile_shift) | sub_tile;
  const uint32_t smbase = sub_tile << a.t;  // swizzled together with the tile index
  const uint32_t ml = a.lo - a.c;
  const uint32_t midlow = tile & ((1u << ml) - 1u);
  const uint32_t hi = tile >> ml;
  const uint32_t cmask = (1u << a.c) - 1u;
  const uint32_t basev = (hi << (a.lo + a.L)) | (midlow << a.c);
  uint32_t x[NQ];

  for (uint32_t k = 0; k < a.K; k++) {
    uint32_t s0, ja, jb;
    if (INV) {
      if (k + 1 < a.K) { s0 = a.c + k * R; ja = 0; jb = R; }
      else { s0 = a.t - R; ja = a.c + k * R - s0; jb = R; }
    } else {
      if (k + 1 < a.K) { s0 = a.t - (k + 1) * R; ja = 0; jb = R; }
      else { s0 = a.c; ja = 0; jb = a.t - k * R - a.c; }
    }
    const uint32_t ebase = ((ltid >> s0) << (s0 + R)) | (ltid & ((1u << s0) - 1u));
    if (k == 0) {
      // the tile's elements are contiguous only when it starts at layer 0
      if (a.vec_ok && s0 == 0 && a.c == 0 && a.lo == 0 && a.src_mask == 0xffffffffu && NQ >= 4) {
        const uint4* p = reinterpret_cast<const uint4*>(src + (basev | ebase));
#pragma unroll
        for (int g = 0; g < NQ / 4; g++) {
          uint4 v = __ldg(p + g);
          x[4 * g] = v.x; x[4 * g + 1] = v.y; x[4 * g + 2] = v.z; x[4 * g + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
          uint32_t e = ebase | ((uint32_t)q << s0);
          uint32_t v = basev | ((e >> a.c) << a.lo) | (e & cmask);
          x[q] = __ldg(src + (v & a.src_mask));
        }
      }
    } else {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < NQ; q++) x[q] = sm[swz(smbase | ebase | ((uint32_t)q << s0))];
      __syncthreads();
    }
    const uint32_t vth = basev | ((ebase >> a.c) << a.lo) | (ebase & cmask);
#pragma unroll
    for (int jj = 0; jj < R; jj++) {
      const int j = INV ? jj : (R - 1 - jj);
      if ((uint32_t)j < ja || (uint32_t)j >= jb) continue;
      const uint32_t i = a.lo + s0 + (uint32_t)j - a.c;
      const uint32_t hth = vth >> (i + 1);
      constexpr int MAXW = NQ / 2;
      uint32_t w[MAXW];
      // COUNT = 2^(R-1-j), resolved at compile time after unrolling
      switch (R - 1 - j) {
        case 0: load_twiddles<1>(w, tw, a.tw_len, a.n, i, hth); break;
        case 1: load_twiddles<2>(w, tw, a.tw_len, a.n, i, hth); break;
        case 2: load_twiddles<4>(w, tw, a.tw_len, a.n, i, hth); break;
        case 3: load_twiddles<8>(w, tw, a.tw_len, a.n, i, hth); break;
        default: load_twiddles<16>(w, tw, a.tw_len, a.n, i, hth); break;
      }
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        if (q & (1 << j)) continue;
        bfly<INV>(x[q], x[q | (1 << j)], w[q >> (j + 1)]);
      }
    }
    if (k + 1 < a.K) {
#pragma unroll
      for (int q = 0; q < NQ; q++) sm[swz(smbase | ebase | ((uint32_t)q << s0))] = x[q];
    } else {
      if (a.has_scale) {
#pragma unroll
        for (int q = 0; q < NQ; q++) x[q] = mul(x[q], a.scale);
      }
      if (a.vec_ok && s0 == 0 && a.c == 0 && a.lo == 0 && NQ >= 4) {
        uint4* p = reinterpret_cast<uint4*>(dst + (basev | ebase));
#pragma unroll
        for (int g = 0; g < NQ / 4; g++) p[g] = make_uint4(x[4 * g], x[4 * g + 1], x[4 * g + 2], x[4 * g + 3]);
      } else {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
          uint32_t e = ebase | ((uint32_t)q << s0);
          uint32_t v = basev | ((e >> a.c) << a.lo) | (e & cmask);
          dst[v] = x[q];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Geometry-specialised pass: the same index mapping as fft_pass_kernel with
// L (layers) and C (contiguous low bits) fixed at compile time, so every
// stage's window, shift and shared-memory offset is a constant:
//  * shared memory is padded (word e at e + e/32) instead of XOR-swizzled;
//    for disjoint bit fields the padding is additive, so the offset of
//    element q folds into the load/store's immediate and each access costs
//    no address arithmetic — and every access pattern of the pass stays
//    bank-conflict free (bank = lane).
// (The adds' pipes: m31.cuh.)
// ---------------------------------------------------------------------------
__host__ __device__ constexpr uint32_t padw(uint32_t e) { return e + (e >> 5); }

template <bool INV, int L, int C>
__global__ void __launch_bounds__(256) fft_tile_kernel(Cols src_tab, MutCols dst_tab,
                                                       const uint32_t* __restrict__ tw, FftPass a) {
  after_previous(src_tab, tw);
  extern __shared__ uint32_t sm[];
  constexpr int R = 5, NQ = 32;
  constexpr int T = L + C;
  constexpr int K = (L + R - 1) / R;
  constexpr int TPT_LOG = T - R;
  constexpr uint32_t CMASK = (1u << C) - 1u;
  const uint32_t col = blockIdx.y;
  const uint32_t* __restrict__ src = src_tab[col];
  uint32_t* __restrict__ dst = dst_tab[col];
  const uint32_t ltid = threadIdx.x & ((1u << TPT_LOG) - 1u);
  const uint32_t sub_tile = threadIdx.x >> TPT_LOG;
  const uint32_t tile = (blockIdx.x << a.tile_shift) | sub_tile;
  const uint32_t ml = a.lo - C;
  const uint32_t midlow = tile & ((1u << ml) - 1u);
  const uint32_t hi = tile >> ml;
  const uint32_t basev = (hi << (a.lo + L)) | (midlow << C);
  const uint32_t tile_pad = padw(sub_tile << T);
  uint32_t x[NQ];

#pragma unroll
  for (int k = 0; k < K; k++) {
    const int s0 = INV ? ((k + 1 < K) ? C + k * R : T - R) : ((k + 1 < K) ? T - (k + 1) * R : C);
    const int ja = INV ? ((k + 1 < K) ? 0 : C + k * R - s0) : 0;
    const int jb = INV ? R : ((k + 1 < K) ? R : T - k * R - C);
    const uint32_t ebase = ((ltid >> s0) << (s0 + R)) | (ltid & ((1u << s0) - 1u));
    const uint32_t pbase = tile_pad + padw(ebase);
    // global offset of element q relative to q = 0 (bits of q << s0 above C
    // move up to the pass's layer bits)
    const uint32_t gbase = basev | ((ebase >> C) << a.lo) | (ebase & CMASK);
    if (k == 0) {
      // contiguous only when the tile starts at layer 0 (C == 0 with lo > 0
      // spaces the elements 2^lo apart)
      if (C == 0 && s0 == 0 && a.lo == 0 && a.vec_ok && a.src_mask == 0xffffffffu) {
        const uint4* p = reinterpret_cast<const uint4*>(src + gbase);
#pragma unroll
        for (int g = 0; g < NQ / 4; g++) {
          uint4 v = __ldg(p + g);
          x[4 * g] = v.x; x[4 * g + 1] = v.y; x[4 * g + 2] = v.z; x[4 * g + 3] = v.w;
        }
      } else {
        // s0 >= C in every stage, so element q sits at gbase + q * 2^(s0-C+lo);
        // with the LDE mask, (gbase | off) & mask = (gbase & mask) + (off & mask)
        const uint32_t* p0 = src + (gbase & a.src_mask);
        const uint32_t stride = 1u << (s0 - C + a.lo);
        if (a.src_mask == 0xffffffffu) {
#pragma unroll
          for (int q = 0; q < NQ; q++) x[q] = __ldg(p0 + (size_t)((uint32_t)q * stride));
        } else {
#pragma unroll
          for (int q = 0; q < NQ; q++) x[q] = __ldg(p0 + (((uint32_t)q * stride) & a.src_mask));
        }
      }
    } else {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < NQ; q++) x[q] = sm[pbase + padw((uint32_t)q << s0)];
      __syncthreads();
    }
#pragma unroll
    for (int jj = 0; jj < R; jj++) {
      const int j = INV ? jj : (R - 1 - jj);
      if (j < ja || j >= jb) continue;
      const uint32_t i = a.lo + (uint32_t)(s0 + j - C);
      const uint32_t hth = gbase >> (i + 1);
      uint32_t w[NQ / 2];
      switch (R - 1 - j) {
        case 0: load_twiddles<1>(w, tw, a.tw_len, a.n, i, hth); break;
        case 1: load_twiddles<2>(w, tw, a.tw_len, a.n, i, hth); break;
        case 2: load_twiddles<4>(w, tw, a.tw_len, a.n, i, hth); break;
        case 3: load_twiddles<8>(w, tw, a.tw_len, a.n, i, hth); break;
        default: load_twiddles<16>(w, tw, a.tw_len, a.n, i, hth); break;
      }
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        if (q & (1 << j)) continue;
        bfly<INV>(x[q], x[q | (1 << j)], w[q >> (j + 1)]);
      }
    }
    if (k + 1 < K) {
#pragma unroll
      for (int q = 0; q < NQ; q++) sm[pbase + padw((uint32_t)q << s0)] = x[q];
    } else {
      if (a.has_scale) {
#pragma unroll
        for (int q = 0; q < NQ; q++) x[q] = mul(x[q], a.scale);
      }
      if (C == 0 && s0 == 0 && a.lo == 0 && a.vec_ok) {
        uint4* p = reinterpret_cast<uint4*>(dst + gbase);
#pragma unroll
        for (int g = 0; g < NQ / 4; g++) p[g] = make_uint4(x[4 * g], x[4 * g + 1], x[4 * g + 2], x[4 * g + 3]);
      } else {
        uint32_t* p0 = dst + gbase;
        const uint32_t stride = 1u << (s0 - C + a.lo);
#pragma unroll
        for (int q = 0; q < NQ; q++) p0[(size_t)((uint32_t)q * stride)] = x[q];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Streaming pass: the passes of large aligned columns. A pass is bound by the
// instructions around its butterflies as much as by the butterflies (7 of
// 11.2 per butterfly in fft_tile_kernel, which reloads, doubles and negates
// its twiddles and forms an address per element for every tile), and its
// warps wait for the tile's loads. So a block fixes the part of the index
// that selects twiddles and walks the columns (and, in a strided pass, the
// tiles) that share it:
//  * the twiddles, centred and doubled for mul_centred, sit in shared memory, built once
//    per block: layer section of size s at [s, 2s), so a thread's 2^k
//    consecutive twiddles are 16-byte shared loads at offsets computed once;
//  * the next tile arrives by 16-byte cp.async while the current one is in its
//    last stage: the buffer is free again once that stage has read it. An
//    evaluation's contiguous pass, which also stores through shared memory
//    (whole lines per warp; its threads end with 32 consecutive words each),
//    has a second buffer for the exchanges and that store, and takes the next
//    tile from the first stage on.
// 2^TB words per tile, 32 per thread (radix 2^5 stages as above). C > 0: a
// strided pass, layers [lo, lo + L) on 2^L rows of 2^C contiguous words, TB =
// L + C. C = 0: layers [0, L) of 2^TB contiguous words (2^(TB - L) transforms).
// Padding, free of bank conflicts in the accesses it serves: e + 4 (e / 128)
// for 16-byte copies and strided stages; e + 4 (e / 32) + 8 (e / 256) where
// threads read and write 32 consecutive words as 16-byte vectors; e + e / 32
// in the second buffer.
// Extension of 158 columns, 2^18 coefficients to 2^20 points: 740 us in 9 + 9
// layers through fft_tile_kernel, 588 us in 8 + 10 here with three reductions
// per butterfly (8.9 against 11.2 instructions), 562 us with two, 553 us with
// stepped addresses in the strided pass; interpolation 198 -> 166 -> 148 us. The extension's memory traffic alone,
// without a butterfly, takes 400 us, the integer ALU pipe's share (4.2
// two-cycle instructions per butterfly, 3 of them in it) 330 us: they overlap
// in part only.
// ---------------------------------------------------------------------------
template <bool INV, int C>
__device__ __host__ constexpr uint32_t in_pad(uint32_t e) {
  return INV && C == 0 ? e + 4 * (e >> 5) + 8 * (e >> 8) : e + 4 * (e >> 7);
}
template <bool INV, int L, int C, int TB>
struct StreamShape {
  static constexpr uint32_t THREADS = 1u << (TB - 5);
  static constexpr bool TWO = !INV && C == 0;  // two buffers
  static constexpr uint32_t IN_WORDS = in_pad<INV, C>(1u << TB);
  static constexpr uint32_t X_WORDS = TWO ? (1u << TB) / 8 * 9 : 0;
  static constexpr uint32_t TW_WORDS = C > 0 ? 1u << L : 1u << (TB - 1);
  static constexpr size_t SMEM = 4 * (size_t)(IN_WORDS + X_WORDS + TW_WORDS);
  // resident blocks: shared memory, and 64 registers per thread with one buffer
  static constexpr int BY_SMEM = (int)((227u << 10) / (SMEM + 1024)), BY_REGS = TWO ? 5 : 1024 / THREADS;
  static constexpr int PER_SM = BY_SMEM < BY_REGS ? BY_SMEM : BY_REGS;
};

// 2^set_log twiddle sets; the `units` tiles of a set (columns x the middle
// index) are walked by `group` blocks. Neighbouring blocks take either the
// sets of one tile position (sets_first: contiguous passes, and an
// extension's first pass, whose replicas then read the coefficients from L2)
// or the tiles of one set (other strided passes: neighbouring rows of memory).
struct StreamGrid {
  uint32_t units, group, set_log, sets_first;
};

template <bool INV, int L, int C, int TB>
__global__ void __launch_bounds__(1 << (TB - 5), (StreamShape<INV, L, C, TB>::PER_SM))
    fft_stream_kernel(Cols src_tab, MutCols dst_tab, const uint32_t* __restrict__ tw, FftPass a, StreamGrid g) {
  after_previous(tw);
  using Shape = StreamShape<INV, L, C, TB>;
  constexpr int R = 5, NQ = 32, T = C > 0 ? TB : L;  // T: tile bits of one transform
  constexpr int K = (L + R - 1) / R;
  constexpr uint32_t THREADS = Shape::THREADS, CMASK = (1u << C) - 1u;
  extern __shared__ uint4 stream_sm[];
  uint32_t* const in = reinterpret_cast<uint32_t*>(stream_sm);
  uint32_t* const ex = Shape::TWO ? in + Shape::IN_WORDS : in;
  uint32_t* const tab = in + Shape::IN_WORDS + Shape::X_WORDS;
  const uint32_t tid = threadIdx.x;
  // C > 0: the high index; C = 0: the chunk of 2^TB words
  const uint32_t set = g.sets_first ? blockIdx.x & ((1u << g.set_log) - 1u) : blockIdx.x / g.group;
  uint32_t unit = g.sets_first ? blockIdx.x >> g.set_log : blockIdx.x - set * g.group;

  // Words of a tile relative to its column; cp.async in 16-byte chunks.
  const uint32_t mid_bits = C > 0 ? a.lo - C : 0;
  auto tile_base = [&](uint32_t u) -> uint32_t {
    return C > 0 ? (set << (a.lo + L)) | ((u & ((1u << mid_bits) - 1u)) << C) : set << TB;
  };
  auto issue = [&](uint32_t u, const uint32_t* src) {
    const uint32_t base = tile_base(u);
    // a strided pass's rows lie below the coefficients' size: the mask cuts the
    // tile's base alone, and the row steps are pointer steps
    const uint32_t e0 = 4 * tid;
    const uint32_t* p = src + ((base & a.src_mask) | ((e0 >> C) << a.lo) | (e0 & CMASK));
    const size_t step = (size_t)(4 * THREADS >> C) << a.lo;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(in + in_pad<INV, C>(4 * tid) + in_pad<INV, C>(4 * THREADS * q));
      if (C == 0) p = src + ((base | (e0 + 4 * THREADS * q)) & a.src_mask);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(p) : "memory");
      if (C > 0) p += step;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  issue(unit, src_tab[unit >> mid_bits]);
  // the next tile's column, one tile ahead of its copies
  const uint32_t* next_src = unit + g.group < g.units ? src_tab[(unit + g.group) >> mid_bits] : nullptr;

  // the block's twiddles, centred and doubled
  if (C > 0) {
    for (uint32_t i = tid; i < (1u << L); i += THREADS) {
      if (i == 0) continue;
      const uint32_t lg = 31 - __clz(i);  // section of 2^lg twiddles: layer lo + L - 1 - lg
      tab[i] = centred2(__ldg(tw + (a.tw_len - (1u << (a.n - a.lo - (L - 1) + lg))) + (set << lg) + (i - (1u << lg))));
    }
  } else {
    // layers 1 .. L - 1; the circle layer 0 takes its twiddles from layer 1's
    for (uint32_t i = tid; i < (1u << (TB - 1)); i += THREADS) {
      if (i < (1u << (TB - L))) continue;
      const uint32_t lg = 31 - __clz(i);  // layer TB - 1 - lg
      tab[i] = centred2(__ldg(tw + (a.tw_len - (1u << (a.n - (TB - 1) + lg))) + (set << lg) + (i - (1u << lg))));
    }
  }

  for (; unit < g.units; unit += g.group) {
    uint32_t* const dst = dst_tab[unit >> mid_bits];
    // the buffer is free: the next tile may arrive
    auto refill = [&] {
      __syncthreads();
      const uint32_t next = unit + g.group;
      if (next < g.units) {
        issue(next, next_src);
        if (next + g.group < g.units) next_src = src_tab[(next + g.group) >> mid_bits];
      }
    };
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the tile has landed (and, the first time, the twiddles)
    uint32_t x[NQ];
#pragma unroll
    for (int k = 0; k < K; k++) {
      // stage windows, as in fft_tile_kernel
      const int s0 = INV ? ((k + 1 < K) ? C + k * R : T - R) : ((k + 1 < K) ? T - (k + 1) * R : C);
      const int ja = INV ? ((k + 1 < K) ? 0 : C + k * R - s0) : 0;
      const int jb = INV ? R : ((k + 1 < K) ? R : T - k * R - C);
      const uint32_t ebase = ((tid >> s0) << (s0 + R)) | (tid & ((1u << s0) - 1u));
      if (k == 0) {
        if (INV && C == 0) {
          const uint4* p = reinterpret_cast<const uint4*>(in + in_pad<INV, C>(ebase));
#pragma unroll
          for (int q = 0; q < NQ / 4; q++) {
            const uint4 v = p[q];
            x[4 * q] = v.x; x[4 * q + 1] = v.y; x[4 * q + 2] = v.z; x[4 * q + 3] = v.w;
          }
        } else {
          const uint32_t* p = in + in_pad<INV, C>(ebase);  // the padding adds over disjoint bit fields
#pragma unroll
          for (int q = 0; q < NQ; q++) x[q] = p[in_pad<INV, C>((uint32_t)q << s0)];
        }
        if (Shape::TWO || K == 1) refill();
      } else {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NQ; q++)
          x[q] = Shape::TWO ? ex[padw(ebase) + padw((uint32_t)q << s0)]
                            : in[in_pad<INV, C>(ebase) + in_pad<INV, C>((uint32_t)q << s0)];
        if (!Shape::TWO && k + 1 == K) refill();
      }
      // twiddle group of this thread's window: its row index above the window
      const uint32_t grp = tid >> s0;
      uint32_t w1[8];  // layer 1's twiddles of this thread, kept for layer 0
#pragma unroll
      for (int jj = 0; jj < R; jj++) {
        const int j = INV ? jj : (R - 1 - jj);
        if (j < ja || j >= jb) continue;
        const int layer = s0 + j - C;           // within the pass
        const int cnt = 1 << (R - 1 - j);       // twiddles per thread
        uint32_t w[NQ / 2];
        if (C == 0 && layer == 0) {
          // s0 = 0: this thread's 16 circle twiddles from its 8 of layer 1
          if (INV || jb == 1) {  // layer 1 comes after, or was in the stage before
            const uint4* p = reinterpret_cast<const uint4*>(tab + (1u << (TB - 2)) + 8 * grp);
            const uint4 u = p[0], v = p[1];
            w1[0] = u.x; w1[1] = u.y; w1[2] = u.z; w1[3] = u.w;
            w1[4] = v.x; w1[5] = v.y; w1[6] = v.z; w1[7] = v.w;
          }
#pragma unroll
          for (int q = 0; q < 4; q++) {  // [y, -y, -x, x]
            w[4 * q] = w1[2 * q + 1];
            w[4 * q + 1] = 0u - w1[2 * q + 1];
            w[4 * q + 2] = 0u - w1[2 * q];
            w[4 * q + 3] = w1[2 * q];
          }
        } else if (C == 0 && layer == 1 && INV) {
#pragma unroll
          for (int q = 0; q < 8; q++) w[q] = w1[q];
        } else {
          // section size: 2^(L - 1 - layer) rows' worth, 2^(TB - 1 - layer) in a contiguous pass
          const uint32_t sec = 1u << ((C > 0 ? L : TB) - 1 - layer);
          const uint32_t* p = tab + sec + (grp << (R - 1 - j));
          if (cnt >= 4) {
#pragma unroll
            for (int q = 0; q < cnt / 4; q++) {
              const uint4 v = reinterpret_cast<const uint4*>(p)[q];
              w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
            }
          } else if (cnt == 2) {
            const uint2 v = *reinterpret_cast<const uint2*>(p);
            w[0] = v.x; w[1] = v.y;
          } else {
            w[0] = *p;
          }
          if (C == 0 && layer == 1 && s0 == 0)
#pragma unroll
            for (int q = 0; q < 8; q++) w1[q] = w[q];
        }
#pragma unroll
        for (int q = 0; q < NQ; q++) {
          if (q & (1 << j)) continue;
          if (INV) bfly_inv(x[q], x[q | (1 << j)], w[q >> (j + 1)]);
          else if (j + 1 < jb && (q >> (j + 1)) & 1) bfly_fwd<true>(x[q], x[q | (1 << j)], w[q >> (j + 1)]);
          else bfly_fwd<false>(x[q], x[q | (1 << j)], w[q >> (j + 1)]);
        }
      }
      // a stage ends with layer j = 0 of its window: signed words go on to the
      // next stage, canonical ones to memory
      if (!INV)
#pragma unroll
        for (int q = 0; q < NQ; q++)
          x[q] = k + 1 == K ? __viaddmin_u32(x[q], q & 1 ? 0u - P : P, x[q]) : q & 1 ? x[q] - P : x[q];
      if (k + 1 < K) {
        if (INV && C == 0 && k == 0) {
          uint4* p = reinterpret_cast<uint4*>(in + in_pad<INV, C>(ebase));
#pragma unroll
          for (int q = 0; q < NQ / 4; q++) p[q] = make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
        } else {
#pragma unroll
          for (int q = 0; q < NQ; q++) {
            if (Shape::TWO) ex[padw(ebase) + padw((uint32_t)q << s0)] = x[q];
            else in[in_pad<INV, C>(ebase) + in_pad<INV, C>((uint32_t)q << s0)] = x[q];
          }
        }
        continue;
      }
      if (INV && a.has_scale) {
        // 1/2^n = 2^(31 - n mod 31): a rotation of the 31-bit word, canonical as it is
#pragma unroll
        for (int q = 0; q < NQ; q++) {
          const uint64_t p = (uint64_t)x[q] * (a.scale << 1);
          x[q] = (uint32_t)(p >> 32) + ((uint32_t)p >> 1);
        }
      }
      if (!INV && C == 0) {
        __syncthreads();  // every thread has read its exchange words
        uint4* o = reinterpret_cast<uint4*>(ex + 36 * tid);  // s0 = 0: row tid of 32 words, 4 of padding
#pragma unroll
        for (int q = 0; q < NQ / 4; q++) o[q] = make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
        __syncthreads();
        uint4* d = reinterpret_cast<uint4*>(dst + (set << TB));
#pragma unroll
        for (int q = 0; q < NQ / 4; q++) {
          const uint32_t e = 4 * tid + 4 * THREADS * q;
          d[tid + THREADS * q] = *reinterpret_cast<const uint4*>(ex + e + 4 * (e >> 5));
        }
      } else if (C > 0) {
        // byte offsets in 32 bits (columns of up to 2^30 words), stepped by a
        // two-input add: 64-bit addresses cost two ALU instructions a word
        uint32_t at = 4u * (tile_base(unit) | ((ebase >> C) << a.lo) | (ebase & CMASK));
        const uint32_t step = 4u << (s0 - C + a.lo);
        char* const d = reinterpret_cast<char*>(dst);
#pragma unroll
        for (int q = 0; q < NQ; q++, at += step) *reinterpret_cast<uint32_t*>(d + at) = x[q];
      } else {
        uint32_t* p0 = dst + (tile_base(unit) | ebase);
#pragma unroll
        for (int q = 0; q < NQ; q++) p0[(size_t)q << s0] = x[q];
      }
    }
  }
}

// Domains of log size 1 and 2: closed forms of cpu/circle.rs:37-60 and
// :193-208, with constants precomputed on the host.
struct SmallFft {
  uint32_t n;
  uint32_t inverse;
  uint32_t k[4];
  uint32_t src_mask;
};
__global__ void fft_small_kernel(Cols src_tab, MutCols dst_tab, SmallFft a, uint32_t n_cols) {
  uint32_t col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= n_cols) return;
  const uint32_t* s = src_tab[col];
  uint32_t* d = dst_tab[col];
  if (a.n == 1) {
    // coefficients beyond 2^coeff_log are zero: these closed forms run every
    // butterfly, so the padding is explicit (the pass kernels skip the copy
    // layers and replicate instead)
    uint32_t v0 = s[0], v1 = 1 <= a.src_mask ? s[1] : 0u;
    if (a.inverse) {  // k = {y_inv, n_inv}
      uint32_t r0 = add(v0, v1), r1 = mul(sub(v0, v1), a.k[0]);
      d[0] = mul(r0, a.k[1]);
      d[1] = mul(r1, a.k[1]);
    } else {  // k = {y}
      uint32_t tmp = mul(v1, a.k[0]);
      d[0] = add(v0, tmp);
      d[1] = sub(v0, tmp);
    }
  } else {
    uint32_t v0 = s[0], v1 = 1 <= a.src_mask ? s[1] : 0u, v2 = 2 <= a.src_mask ? s[2] : 0u,
             v3 = 3 <= a.src_mask ? s[3] : 0u;
    if (a.inverse) {  // k = {x_inv, y_inv, n_inv}
      auto ib = [](uint32_t& p, uint32_t& q, uint32_t w) { uint32_t t0 = p; p = add(t0, q); q = mul(sub(t0, q), w); };
      ib(v0, v1, a.k[1]);
      ib(v2, v3, neg(a.k[1]));
      ib(v0, v2, a.k[0]);
      ib(v1, v3, a.k[0]);
      d[0] = mul(v0, a.k[2]); d[1] = mul(v1, a.k[2]); d[2] = mul(v2, a.k[2]); d[3] = mul(v3, a.k[2]);
    } else {  // k = {x, y}
      auto fb = [](uint32_t& p, uint32_t& q, uint32_t w) { uint32_t t0 = mul(q, w); q = sub(p, t0); p = add(p, t0); };
      fb(v0, v2, a.k[0]);
      fb(v1, v3, a.k[0]);
      fb(v0, v1, a.k[1]);
      fb(v2, v3, neg(a.k[1]));
      d[0] = v0; d[1] = v1; d[2] = v2; d[3] = v3;
    }
  }
}

// Host-side circle point at a circle index (double-and-add on the host).
static pt31 host_index_to_point(uint32_t k) {
  pt31 r = {1u, 0u}, cur = {2u, 1268011823u};
  for (int b = 0; b < 31; b++) {
    if ((k >> b) & 1u) r = pt_add(r, cur);
    cur = pt_add(cur, cur);
  }
  return r;
}
// Initial point of the half coset of CanonicCoset(n): index 2^(31 - (n + 1)).
static pt31 canonic_half_coset_initial(uint32_t n) { return host_index_to_point(1u << (31 - (n + 1))); }

static int launch_small(cudaStream_t st, Cols src, MutCols dst, uint32_t n_cols, uint32_t n,
                        bool inverse, uint32_t src_mask) {
  pt31 p = canonic_half_coset_initial(n);
  SmallFft a{};
  a.n = n;
  a.inverse = inverse;
  a.src_mask = src_mask;
  if (n == 1) {
    if (inverse) {
      uint32_t yn_inv = inv(mul(p.y, 2));
      a.k[0] = mul(yn_inv, 2);     // y_inv
      a.k[1] = mul(yn_inv, p.y);   // n_inv
    } else {
      a.k[0] = p.y;
    }
  } else {
    if (inverse) {
      uint32_t xyn_inv = inv(mul(mul(p.x, p.y), 4));
      a.k[0] = mul(mul(xyn_inv, p.y), 4);  // x_inv
      a.k[1] = mul(mul(xyn_inv, p.x), 4);  // y_inv
      a.k[2] = mul(mul(xyn_inv, p.x), p.y);  // n_inv
    } else {
      a.k[0] = p.x;
      a.k[1] = p.y;
    }
  }
  uint32_t threads = 128;
  fft_small_kernel<<<(n_cols + threads - 1) / threads, threads, 0, st>>>(src, dst, a, n_cols);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}

struct FftTuning {
  uint32_t tile_log;       // log2 of the shared-memory tile (elements), <= 13; 0: by size
  uint32_t coalesce_bits;  // contiguous low bits per strided tile row
};
// Per number of computed layers (an FFT of 2^n, or an LDE from 2^n
// coefficients, computes n layers) and extension (domain log size minus
// layers: 0 for an FFT, the blowup for an LDE; capped at FFT_MAX_EXT). Written
// at set-up (set_fft_tuning, fft_autotune, reset_fft_tuning), read by every
// launch. Zero, as at the start: the split by size.
constexpr uint32_t FFT_MAX_EXT = 3;
static FftTuning g_fft_tuning[32][FFT_MAX_EXT + 1];
static void split_layers(uint32_t layers, FftTuning tn, std::vector<std::pair<uint32_t, uint32_t>>& parts);

// The split by size, within tiles of 2^13. Fewest passes, then fewest register
// stages (of up to 5 layers), then the wider rows of 12/5 (whole 128-byte
// lines). 13/4, whose strided passes hold 9 layers in tiles of 2^13, only where
// it saves a pass. 158 columns of 2^18: 9 + 9 layers (13/4) 167 us interpolated
// and 306 extended by 1, 10 + 8 (12/4) 159 and 292; 17 layers of 128 columns,
// 10 + 7 against 8 + 9, 63 against 72. Over 13..24 layers of 1 to 256 columns,
// extended by 0 to 2, it is within 8% of the best of 13/4, 12/4, 12/5, 13/5,
// 11/5 and 10/4, at nine shapes in ten within 3%, except at 22 layers of few
// columns, where its two passes take 1.03 to 1.11 times as long as three. 13/4
// at every size takes up to 1.19 times as long.
static FftTuning split_by_size(uint32_t layers) {
  FftTuning best{13, 4};
  size_t best_passes = 99, best_stages = 0;
  for (FftTuning tn : {FftTuning{12, 5}, FftTuning{12, 4}, FftTuning{13, 4}}) {
    std::vector<std::pair<uint32_t, uint32_t>> parts;
    split_layers(layers, tn, parts);
    size_t stages = 0;
    for (auto& p : parts) stages += (p.second + 4) / 5;
    if (parts.size() < best_passes || (parts.size() == best_passes && tn.tile_log == 12 && stages < best_stages)) {
      best = tn;
      best_passes = parts.size();
      best_stages = stages;
    }
  }
  return best;
}
struct SplitsBySize {
  FftTuning of[32];
  SplitsBySize() {
    for (uint32_t l = 0; l < 32; l++) of[l] = split_by_size(l);
  }
};
static uint32_t ext_slot(uint32_t layers, uint32_t n) {
  return n - layers < FFT_MAX_EXT ? n - layers : FFT_MAX_EXT;
}
static FftTuning tuning_for(uint32_t layers, uint32_t n) {
  static const SplitsBySize by_size;
  const uint32_t l = layers < 32 ? layers : 31;
  const FftTuning t = g_fft_tuning[l][ext_slot(layers, n)];
  return t.tile_log ? t : by_size.of[l];
}
// An entry as it is read back: 13/4 where nothing was installed.
static FftTuning reported(FftTuning t) { return t.tile_log ? t : FftTuning{13, 4}; }

// Splits layers [0, layers) into balanced passes (lo, L): the first pass has
// the whole tile for layers, later ones reserve `coalesce_bits` of it.
static void split_layers(uint32_t layers, FftTuning tn, std::vector<std::pair<uint32_t, uint32_t>>& parts) {
  const uint32_t T = tn.tile_log, C = tn.coalesce_bits;
  if (layers <= T) {
    parts.push_back({0, layers});
    return;
  }
  uint32_t np = 1 + (layers - T + (T - C) - 1) / (T - C);
  uint32_t lr = std::min(T - C, (layers + np - 1) / np);
  uint32_t l0 = layers - lr * (np - 1);
  parts.push_back({0, l0});
  uint32_t lo = l0;
  for (uint32_t p = 1; p < np; p++) {
    parts.push_back({lo, lr});
    lo += lr;
  }
}

static void fft_partition(uint32_t layers, uint32_t n, std::vector<std::pair<uint32_t, uint32_t>>& parts) {
  split_layers(layers, tuning_for(layers, n), parts);
}

template <bool INV, int R>
static void launch_pass(cudaStream_t st, dim3 grid, uint32_t threads, size_t smem, Cols s,
                        MutCols d, const uint32_t* tw, const FftPass& a) {
  fft_pass_kernel<INV, R><<<grid, threads, smem, st>>>(s, d, tw, a);
  note_launch();
}

template <bool INV, int L, int C>
static void launch_tile(cudaStream_t st, dim3 grid, uint32_t threads, Cols s, MutCols d,
                        const uint32_t* tw, const FftPass& a) {
  const uint32_t words = 1u << (a.t + a.tile_shift);
  const size_t smem = (size_t)4 * (words + (words >> 5));
  launch_after(fft_tile_kernel<INV, L, C>, grid, threads, smem, st, s, d, tw, a);
  note_launch();
}

// GS_FFT_GENERIC=1 forces the generic pass (for comparisons).
static bool fft_generic() {
  static const bool generic = [] {
    const char* e = getenv("GS_FFT_GENERIC");
    return e && e[0] == '1';
  }();
  return generic;
}

// Tiles per block: the chip's share of all tiles in whole waves of equal
// blocks, each of 8 tiles or a few more (one wave below 16; 4 tiles against 5
// in a wave and a bit took 35 us against 26 on 100 columns of 2^17), at most
// a set's.
static uint32_t stream_tiles(uint32_t set_log, uint32_t units, uint32_t per_sm) {
  const uint64_t resident = (uint64_t)num_sms() * per_sm, total = (uint64_t)units << set_log;
  const uint64_t waves = std::max<uint64_t>(1, total / (8 * resident));
  return (uint32_t)std::min<uint64_t>(units, (total + waves * resident - 1) / (waves * resident));
}

template <bool INV, int L, int C, int TB>
static int launch_stream(cudaStream_t st, uint32_t n_cols, Cols s, MutCols d,
                         const uint32_t* tw, const FftPass& a) {
  using Shape = StreamShape<INV, L, C, TB>;
  static OncePerDevice smem;
  GS_CUDA_TRY(allow_smem(smem, fft_stream_kernel<INV, L, C, TB>, Shape::SMEM));
  StreamGrid g;
  g.set_log = C > 0 ? a.n - a.lo - L : a.n - TB;
  g.units = C > 0 ? n_cols << (a.lo - C) : n_cols;
  g.sets_first = C == 0 || a.src_mask != 0xffffffffu;
  const uint32_t per = stream_tiles(g.set_log, g.units, Shape::PER_SM);
  g.group = (g.units + per - 1) / per;
  launch_after(fft_stream_kernel<INV, L, C, TB>, g.group << g.set_log, Shape::THREADS, Shape::SMEM, st, s, d, tw, a, g);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}

// Passes the streaming kernel takes: aligned columns of at least one tile,
// contiguous passes of 5..13 layers, strided ones of 5..9 whose rows of
// 2^(TB - L) words start a layer range high enough. *taken says whether it ran.
// A contiguous pass builds a table of half a tile's words per block, which
// takes 4 tiles to pay (one column of 2^24, a tile per block: 46 -> 77 us).
constexpr uint32_t STREAM_MIN_TILES = 4;
// Without `launch` it only says so.
template <bool INV>
static int launch_stream_any(cudaStream_t st, uint32_t n_cols, Cols s, MutCols d,
                             const uint32_t* tw, const FftPass& a, bool* taken, bool launch = true) {
  *taken = false;
  if (fft_generic() || !a.vec_ok || (uint64_t)n_cols << a.n >= 1ull << 40) return OK;
#define GS_STREAM(LL, CC, TB)                                                   \
  case LL:                                                                      \
    if (a.n < TB || (CC > 0 && a.lo < CC)) return OK;                           \
    if (CC == 0 && stream_tiles(a.n - TB, n_cols, StreamShape<INV, LL, CC, TB>::PER_SM) < STREAM_MIN_TILES) \
      return OK;                                                                \
    *taken = true;                                                              \
    return launch ? launch_stream<INV, LL, CC, TB>(st, n_cols, s, d, tw, a) : OK;
  if (a.lo == 0) {
    switch (a.L) { GS_STREAM(5, 0, 12) GS_STREAM(6, 0, 12) GS_STREAM(7, 0, 12) GS_STREAM(8, 0, 12) GS_STREAM(9, 0, 12)
                   GS_STREAM(10, 0, 12) GS_STREAM(11, 0, 12) GS_STREAM(12, 0, 12) GS_STREAM(13, 0, 13)
                   default: return OK; }
  }
  switch (a.L) { GS_STREAM(5, 7, 12) GS_STREAM(6, 6, 12) GS_STREAM(7, 5, 12) GS_STREAM(8, 4, 12) GS_STREAM(9, 4, 13)
                 default: return OK; }
#undef GS_STREAM
}

// The specialised kernel covers first passes (C = 0, 5..13 layers) and later
// passes with 16 or 32 contiguous words per tile row (C = 4 with 5..9 layers,
// C = 5 with 5..8); anything else runs the generic pass. Without `launch` it
// only says which.
template <bool INV>
static bool launch_tile_any(cudaStream_t st, dim3 grid, uint32_t threads, Cols s,
                            MutCols d, const uint32_t* tw, const FftPass& a, bool launch = true) {
  if (fft_generic()) return false;
#define GS_TILE(LL, CC)                                                   \
  case LL:                                                                \
    if (launch) launch_tile<INV, LL, CC>(st, grid, threads, s, d, tw, a); \
    return true;
  if (a.c == 0) {
    switch (a.L) { GS_TILE(5, 0) GS_TILE(6, 0) GS_TILE(7, 0) GS_TILE(8, 0) GS_TILE(9, 0) GS_TILE(10, 0)
                   GS_TILE(11, 0) GS_TILE(12, 0) GS_TILE(13, 0) default: return false; }
  }
  if (a.c == 4) {
    switch (a.L) { GS_TILE(5, 4) GS_TILE(6, 4) GS_TILE(7, 4) GS_TILE(8, 4) GS_TILE(9, 4) default: return false; }
  }
  if (a.c == 5) {
    switch (a.L) { GS_TILE(5, 5) GS_TILE(6, 5) GS_TILE(7, 5) GS_TILE(8, 5) default: return false; }
  }
#undef GS_TILE
  return false;
}

// Column pointers of the current call are 16-byte aligned (checked by the
// callers that know them on the host; a device table is opaque here).
static thread_local bool g_cols_aligned = true;
void fft_set_columns_aligned(bool aligned) { g_cols_aligned = aligned; }

template <bool INV>
static FftPass pass_of(uint32_t n, uint32_t layers, std::pair<uint32_t, uint32_t> part, bool first, bool last,
                       uint32_t src_mask, uint32_t tw_len, bool aligned) {
  FftPass a{};
  a.n = n;
  a.lo = part.first;
  a.L = part.second;
  a.c = std::min(tuning_for(layers, n).coalesce_bits, a.lo);
  a.t = a.c + a.L;
  const uint32_t R = std::min<uint32_t>(5, a.L);
  a.K = (a.L + R - 1) / R;
  a.src_mask = first ? src_mask : 0xffffffffu;
  a.tw_len = tw_len;
  a.has_scale = (INV && last) ? 1u : 0u;
  a.scale = a.has_scale ? inv(1u << n) : 1u;
  a.vec_ok = aligned ? 1u : 0u;
  const uint32_t tpt_log = a.t - R, tiles_log = n - a.t;
  a.tile_shift = std::min(tpt_log < 7 ? 7 - tpt_log : 0u, tiles_log);
  return a;
}

template <bool INV>
static int run_passes(cudaStream_t st, Cols src, MutCols dst, uint32_t n_cols, uint32_t n,
                      uint32_t layers, uint32_t src_mask, const uint32_t* tw, uint32_t tw_len) {
  std::vector<std::pair<uint32_t, uint32_t>> parts;
  fft_partition(layers, n, parts);
  if (!INV) std::reverse(parts.begin(), parts.end());
  for (size_t p = 0; p < parts.size(); p++) {
    const FftPass a = pass_of<INV>(n, layers, parts[p], p == 0, p + 1 == parts.size(), src_mask, tw_len, g_cols_aligned);
    const uint32_t R = std::min<uint32_t>(5, a.L), tile_shift = a.tile_shift;
    const uint32_t tiles_log = n - a.t;
    const uint32_t threads = 1u << (a.t - R + tile_shift);
    const size_t smem = (size_t)4 << (a.t + tile_shift);
    dim3 grid(1u << (tiles_log - tile_shift), n_cols);
    Cols s = (p == 0) ? src : Cols(dst);
    bool taken = false;
    GS_TRY(launch_stream_any<INV>(st, n_cols, s, dst, tw, a, &taken));
    if (taken) continue;
    if (R == 5 && launch_tile_any<INV>(st, grid, threads, s, dst, tw, a)) {
      GS_CUDA_TRY(cudaGetLastError());
      continue;
    }
    switch (R) {
      case 1: launch_pass<INV, 1>(st, grid, threads, smem, s, dst, tw, a); break;
      case 2: launch_pass<INV, 2>(st, grid, threads, smem, s, dst, tw, a); break;
      case 3: launch_pass<INV, 3>(st, grid, threads, smem, s, dst, tw, a); break;
      case 4: launch_pass<INV, 4>(st, grid, threads, smem, s, dst, tw, a); break;
      default: launch_pass<INV, 5>(st, grid, threads, smem, s, dst, tw, a); break;
    }
    GS_CUDA_TRY(cudaGetLastError());
  }
  return OK;
}

// The passes of an FFT of n_cols aligned columns, in the order of launch: first
// layer, layers, kernel (0 generic, 1 a tile per block, 2 streaming).
template <bool INV>
static void list_passes(uint32_t n, uint32_t layers, uint32_t n_cols, uint32_t* out, uint32_t* n_out) {
  std::vector<std::pair<uint32_t, uint32_t>> parts;
  fft_partition(layers, n, parts);
  if (!INV) std::reverse(parts.begin(), parts.end());
  for (size_t p = 0; p < parts.size(); p++) {
    const FftPass a = pass_of<INV>(n, layers, parts[p], p == 0, p + 1 == parts.size(),
                                   layers == n ? 0xffffffffu : (1u << layers) - 1u, 1u << (n - 1), true);
    bool streams = false;
    (void)launch_stream_any<INV>(nullptr, n_cols, Cols(), MutCols(), nullptr, a, &streams, false);
    const bool tile = a.L >= 5 && launch_tile_any<INV>(nullptr, dim3(), 0, Cols(), MutCols(), nullptr, a, false);
    out[3 * p] = a.lo;
    out[3 * p + 1] = a.L;
    out[3 * p + 2] = streams ? 2u : tile ? 1u : 0u;
  }
  *n_out = (uint32_t)parts.size();
}
int fft_passes(uint32_t log_n, uint32_t coeff_log, uint32_t n_cols, bool inverse, uint32_t* out, uint32_t* n_out) {
  GS_REQUIRE(log_n >= 1 && log_n <= 30 && coeff_log >= 1 && coeff_log <= log_n, "log size out of range");
  GS_REQUIRE(n_cols >= 1 && n_cols <= 65535, "number of columns out of range");
  GS_REQUIRE(!inverse || coeff_log == log_n, "an interpolation computes every layer");
  GS_REQUIRE(out && n_out, "null output");
  *n_out = 0;
  if (log_n <= 2) return OK;  // closed forms
  if (inverse) list_passes<true>(log_n, coeff_log, n_cols, out, n_out);
  else list_passes<false>(log_n, coeff_log, n_cols, out, n_out);
  return OK;
}

int interpolate_columns(cudaStream_t st, MutCols d_cols, uint32_t n_cols, uint32_t log_n,
                        const uint32_t* d_itwiddles, uint32_t tw_log) {
  if (n_cols == 0) return OK;
  GS_REQUIRE(log_n >= 1 && log_n <= 30, "log_n out of range");
  GS_REQUIRE(n_cols <= 65535, "too many columns in one call");
  if (log_n <= 2) return launch_small(st, d_cols, d_cols, n_cols, log_n, true, 0xffffffffu);
  GS_REQUIRE(tw_log + 1 >= log_n, "twiddle tree too small for the domain");
  return run_passes<true>(st, d_cols, d_cols, n_cols, log_n, log_n, 0xffffffffu, d_itwiddles,
                          1u << tw_log);
}

// Out-of-place interpolation (src and dst tables may differ).
int interpolate_columns_to(cudaStream_t st, Cols d_src, MutCols d_dst, uint32_t n_cols,
                           uint32_t log_n, const uint32_t* d_itwiddles, uint32_t tw_log) {
  if (n_cols == 0) return OK;
  GS_REQUIRE(log_n >= 1 && log_n <= 30, "log_n out of range");
  GS_REQUIRE(n_cols <= 65535, "too many columns in one call");
  if (log_n <= 2) return launch_small(st, d_src, d_dst, n_cols, log_n, true, 0xffffffffu);
  GS_REQUIRE(tw_log + 1 >= log_n, "twiddle tree too small for the domain");
  return run_passes<true>(st, d_src, d_dst, n_cols, log_n, log_n, 0xffffffffu, d_itwiddles, 1u << tw_log);
}

int evaluate_columns(cudaStream_t st, Cols d_src, uint32_t coeff_log, MutCols d_dst,
                     uint32_t n_cols, uint32_t log_n, const uint32_t* d_twiddles, uint32_t tw_log) {
  if (n_cols == 0) return OK;
  GS_REQUIRE(log_n >= 1 && log_n <= 30, "log_n out of range");
  GS_REQUIRE(coeff_log >= 1 && coeff_log <= log_n, "coefficient log size must be in [1, log_n]");
  GS_REQUIRE(n_cols <= 65535, "too many columns in one call");
  uint32_t src_mask = (1u << coeff_log) - 1u;
  if (log_n <= 2) return launch_small(st, d_src, d_dst, n_cols, log_n, false, src_mask);
  GS_REQUIRE(tw_log + 1 >= log_n, "twiddle tree too small for the domain");
  return run_passes<false>(st, d_src, d_dst, n_cols, log_n, coeff_log, src_mask, d_twiddles, 1u << tw_log);
}

// ------------------------------------------------------------- work-list
// Device form of an item: the host adds the 1/2^log scale of an
// interpolation.
struct FftWlItem {
  const uint32_t* src;
  uint32_t* dst;
  uint32_t log, coeff_log, inverse, scale;
};

// Persistent grid: block b takes items b, b + gridDim.x, ... of a list sorted
// by decreasing size, so the large items start first. Each item runs whole in
// shared memory: load (an evaluation replicates its 2^coeff_log
// coefficients over the domain, the top layers of the zero-padded FFT being
// copies), the layers with the twiddle rule of the pass kernels (line layer
// i >= 1: tw[tw_len - 2^(log - i) + h]; circle layer 0: circle_twiddle), one
// block barrier per layer, then the store (scaled for an interpolation).
__global__ void __launch_bounds__(256) fft_worklist_kernel(const FftWlItem* __restrict__ items, uint32_t n_items,
                                                           const uint32_t* __restrict__ tw,
                                                           const uint32_t* __restrict__ itw, uint32_t tw_len) {
  extern __shared__ uint32_t sm[];
  for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {
    const FftWlItem w = items[it];
    const uint32_t n = w.log, N = 1u << n;
    const uint32_t cmask = w.inverse ? N - 1u : (1u << w.coeff_log) - 1u;
    for (uint32_t v = threadIdx.x; v < N; v += blockDim.x) sm[v] = __ldg(w.src + (v & cmask));
    __syncthreads();
    const uint32_t* t = w.inverse ? itw : tw;
    const uint32_t layers = w.inverse ? n : w.coeff_log;
    for (uint32_t k = 0; k < layers; k++) {
      const uint32_t i = w.inverse ? k : layers - 1 - k;
      for (uint32_t j = threadIdx.x; j < N / 2; j += blockDim.x) {
        const uint32_t h = j >> i;
        const uint32_t v = (h << (i + 1)) | (j & ((1u << i) - 1u));
        const uint32_t u = v + (1u << i);
        const uint32_t tw_h = i == 0 ? circle_twiddle(t, tw_len, n, h) : __ldg(t + tw_len - (1u << (n - i)) + h);
        const uint32_t a = sm[v], b = sm[u];
        if (w.inverse) {
          sm[v] = add(a, b);
          sm[u] = mul(sub(a, b), tw_h);
        } else {
          const uint32_t p = mul(b, tw_h);
          sm[v] = add(a, p);
          sm[u] = sub(a, p);
        }
      }
      __syncthreads();
    }
    for (uint32_t v = threadIdx.x; v < N; v += blockDim.x) w.dst[v] = w.inverse ? mul(sm[v], w.scale) : sm[v];
    __syncthreads();  // the next item reuses the shared buffer
  }
}

int fft_worklist(Context& ctx, const FftItem* items, uint32_t n_items, const uint32_t* d_twiddles,
                 const uint32_t* d_itwiddles, uint32_t tw_log) {
  if (n_items == 0) return OK;
  GS_REQUIRE(items != nullptr, "null item list");
  GS_REQUIRE(tw_log <= 30, "twiddle log size out of range");
  cudaStream_t st = ctx.stream;
  // 1/2^log for every log, once; the items bucketed by size, largest first
  static const std::vector<uint32_t> inv_pow2 = [] {
    std::vector<uint32_t> t(31);
    for (uint32_t k = 0; k <= 30; k++) t[k] = inv(1u << k);
    return t;
  }();
  uint32_t count[FFT_WL_MAX_LOG + 1] = {0};
  for (uint32_t k = 0; k < n_items; k++) {
    const FftItem& x = items[k];
    GS_REQUIRE(x.src && x.dst, "null column in a work-list item");
    GS_REQUIRE(x.log >= 1 && x.log <= 30 && tw_log + 1 >= x.log, "work-list item size out of range");
    GS_REQUIRE(x.inverse || (x.coeff_log >= 1 && x.coeff_log <= x.log), "coefficient log size must be in [1, log]");
    GS_REQUIRE(x.inverse ? d_itwiddles != nullptr : d_twiddles != nullptr, "null twiddle tree");
    if (x.log >= FFT_WL_MIN_LOG && x.log <= FFT_WL_MAX_LOG) count[x.log]++;
  }
  uint32_t first[FFT_WL_MAX_LOG + 2] = {0}, total = 0;
  for (int lg = (int)FFT_WL_MAX_LOG; lg >= (int)FFT_WL_MIN_LOG; lg--) {
    first[lg] = total;
    total += count[lg];
  }
  std::vector<FftWlItem> wl(total);
  for (uint32_t k = 0; k < n_items; k++) {
    const FftItem& x = items[k];
    if (x.log < FFT_WL_MIN_LOG || x.log > FFT_WL_MAX_LOG) continue;
    wl[first[x.log]++] = FftWlItem{x.src, x.dst, x.log, x.inverse ? x.log : x.coeff_log, x.inverse ? 1u : 0u,
                                   x.inverse ? inv_pow2[x.log] : 1u};
  }
  // the items outside the shared-memory range, one call each
  for (uint32_t k = 0; k < n_items; k++) {
    const FftItem& x = items[k];
    if (x.log >= FFT_WL_MIN_LOG && x.log <= FFT_WL_MAX_LOG) continue;
    if (x.inverse)
      GS_TRY(interpolate_columns_to(st, Cols(x.src, 0), MutCols(x.dst, 0), 1, x.log, d_itwiddles, tw_log));
    else
      GS_TRY(evaluate_columns(st, Cols(x.src, 0), x.coeff_log, MutCols(x.dst, 0), 1, x.log, d_twiddles, tw_log));
  }
  if (wl.empty()) return OK;
  const void* d = nullptr;
  void* owned = nullptr;  // a list too long for the staging ring: a buffer of its own
  const size_t bytes = wl.size() * sizeof(FftWlItem);
  if (bytes <= ctx.ring_cap / 2) {
    GS_TRY(ctx.stage_bytes(wl.data(), bytes, &d));
  } else {
    GS_TRY(ctx.alloc_async(bytes, &owned));
    GS_CUDA_TRY(cudaMemcpyAsync(owned, wl.data(), bytes, cudaMemcpyHostToDevice, st));
    d = owned;
  }
  const size_t smem = (size_t)4 << wl.front().log;
  static OncePerDevice limit;
  GS_CUDA_TRY(allow_smem(limit, fft_worklist_kernel, (size_t)4 << FFT_WL_MAX_LOG));
  const uint32_t per_sm = (uint32_t)std::min<size_t>(8, (200u << 10) / smem);
  const uint32_t grid = (uint32_t)std::min<size_t>(wl.size(), (size_t)num_sms() * (per_sm ? per_sm : 1));
  fft_worklist_kernel<<<grid, 256, smem, st>>>((const FftWlItem*)d, (uint32_t)wl.size(), d_twiddles, d_itwiddles,
                                               1u << tw_log);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  if (owned) GS_CUDA_TRY(cudaFreeAsync(owned, st));  // stream-ordered: after the kernel
  return OK;
}

// Installs the tuning for FFTs computing `layers` layers (0: every size) on
// a domain `ext` log sizes larger (ext > FFT_MAX_EXT: every extension). A
// tile holds 2^tile_log words (at most 2^13, 32 KiB of shared memory), of
// which 2^coalesce_bits are contiguous in memory; a pass needs room for 5
// layers besides them.
int set_fft_tuning(uint32_t layers, uint32_t ext, uint32_t tile_log, uint32_t coalesce_bits) {
  GS_REQUIRE(layers < 32, "log size out of range");
  GS_REQUIRE(tile_log >= 6 && tile_log <= 13, "tile log must be in [6, 13]");
  GS_REQUIRE(coalesce_bits <= 5 && coalesce_bits + 5 <= tile_log, "coalesced bits must be <= min(5, tile_log - 5)");
  for (uint32_t l = layers; l < (layers ? layers + 1 : 32u); l++)
    for (uint32_t e = 0; e <= FFT_MAX_EXT; e++)
      if (ext > FFT_MAX_EXT || e == ext) g_fft_tuning[l][e] = FftTuning{tile_log, coalesce_bits};
  return OK;
}

void reset_fft_tuning() {
  for (auto& row : g_fft_tuning)
    for (FftTuning& t : row) t = FftTuning{0, 0};
}

// Picks, for every FFT log size n in [lo, hi] and extension e in [0,
// max_ext], the tile size and coalesced row width whose pass split is
// fastest, and installs it. e = 0 times an evaluate + interpolate round trip
// of 2^n-word columns in place; e > 0 an LDE of 2^n coefficients onto 2^(n+e)
// points, the shape of a commitment's or constraint domain's extension.
// Scratch columns fill 2^24 output words (or one column when larger); sizes
// whose output exceeds the scratch keep their tuning. Each split is timed with
// CUDA events as the best of 3 trials of 3 runs; the installed split (first
// in the list) is replaced only by one at least 2% faster, so timing noise
// does not move it; the split by size, where it stays, is installed as what it
// is. Candidates that give the same pass split as an earlier
// one are not timed again. Every candidate computes the same values; only the
// split, and so the speed, differ. Not thread-safe against concurrent
// launches (a set-up step). Outputs: (hi - lo + 1) x (max_ext + 1), by size.
int fft_autotune(cudaStream_t st, uint32_t lo, uint32_t hi, uint32_t max_ext, const uint32_t* tw, const uint32_t* itw,
                 uint32_t tw_log, uint32_t* out_tile, uint32_t* out_coalesce) {
  GS_REQUIRE(lo >= 3 && hi <= 27 && lo <= hi && max_ext <= FFT_MAX_EXT && tw_log + 1 >= hi,
             "autotune range out of bounds");
  static const FftTuning fixed[] = {{13, 4}, {12, 4}, {11, 4}, {10, 4}, {13, 5}, {12, 5}, {11, 5}, {13, 3}};
  const uint32_t w_log = hi > 24 ? hi : 24;
  const size_t words = (size_t)1 << w_log;
  uint32_t* buf = nullptr;  // outputs (and in-place round trips)
  uint32_t* src = nullptr;  // LDE inputs
  uint32_t** tab = nullptr;
  uint32_t** stab = nullptr;
  const uint32_t max_cols = 32768;
  GS_CUDA_TRY(cudaMallocAsync((void**)&buf, 4 * words, st));
  GS_CUDA_TRY(cudaMallocAsync((void**)&src, 2 * words, st));
  GS_CUDA_TRY(cudaMallocAsync((void**)&tab, sizeof(void*) * max_cols, st));
  GS_CUDA_TRY(cudaMallocAsync((void**)&stab, sizeof(void*) * max_cols, st));
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int rc = OK;
  if (cudaMemsetAsync(buf, 0, 4 * words, st) != cudaSuccess || cudaMemsetAsync(src, 0, 2 * words, st) != cudaSuccess ||
      cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)
    rc = ERR_CUDA;
  const bool aligned = g_cols_aligned;
  g_cols_aligned = true;
  std::vector<uint32_t*> h, hs;
  for (uint32_t n = lo; n <= hi && rc == OK; n++) {
    for (uint32_t e = 0; e <= max_ext && rc == OK; e++) {
      const uint32_t dn = n + e;  // domain log size
      const size_t slot = (size_t)(n - lo) * (max_ext + 1) + e;
      if (dn > w_log || tw_log + 1 < dn) {
        if (out_tile) out_tile[slot] = reported(g_fft_tuning[n][e]).tile_log;
        if (out_coalesce) out_coalesce[slot] = reported(g_fft_tuning[n][e]).coalesce_bits;
        continue;
      }
      const uint32_t cols = (uint32_t)std::min<size_t>(words >> dn, max_cols);
      h.resize(cols);
      hs.resize(cols);
      for (uint32_t c = 0; c < cols; c++) {
        h[c] = buf + ((size_t)c << dn);
        hs[c] = src + ((size_t)c << n);
      }
      if (cudaMemcpyAsync(tab, h.data(), sizeof(void*) * cols, cudaMemcpyHostToDevice, st) != cudaSuccess ||
          cudaMemcpyAsync(stab, hs.data(), sizeof(void*) * cols, cudaMemcpyHostToDevice, st) != cudaSuccess ||
          cudaStreamSynchronize(st) != cudaSuccess) {
        rc = ERR_CUDA;
        break;
      }
      const FftTuning before = g_fft_tuning[n][e], keep = tuning_for(n, dn);
      float best = 1e30f, keep_ms = 1e30f;
      FftTuning pick = keep;
      std::vector<std::vector<std::pair<uint32_t, uint32_t>>> seen;
      std::vector<FftTuning> cand(1, keep);
      cand.insert(cand.end(), std::begin(fixed), std::end(fixed));
      for (size_t ci = 0; ci < cand.size() && rc == OK; ci++) {
        const FftTuning c = cand[ci];
        g_fft_tuning[n][e] = c;
        std::vector<std::pair<uint32_t, uint32_t>> parts;
        fft_partition(n, dn, parts);
        for (auto& pr : parts) pr.first = std::min(c.coalesce_bits, pr.first) | (pr.first << 8);
        if (std::find(seen.begin(), seen.end(), parts) != seen.end()) continue;
        seen.push_back(parts);
        float ms = 1e30f;
        for (int trial = 0; trial < 4 && rc == OK; trial++) {  // trial 0 warms up
          for (int rep = 0; rep < 3 && rc == OK; rep++) {
            if (rep == 0 && cudaEventRecord(e0, st) != cudaSuccess) rc = ERR_CUDA;
            if (rc != OK) break;
            if (e == 0) {
              rc = run_passes<false>(st, (const uint32_t* const*)tab, tab, cols, n, n, 0xffffffffu, tw, 1u << tw_log);
              if (rc == OK)
                rc = run_passes<true>(st, (const uint32_t* const*)tab, tab, cols, n, n, 0xffffffffu, itw,
                                      1u << tw_log);
            } else {
              rc = run_passes<false>(st, (const uint32_t* const*)stab, tab, cols, dn, n, (1u << n) - 1u, tw,
                                     1u << tw_log);
            }
          }
          float t = 0;
          if (rc == OK && (cudaEventRecord(e1, st) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
                           cudaEventElapsedTime(&t, e0, e1) != cudaSuccess))
            rc = ERR_CUDA;
          if (rc == OK && trial > 0) ms = std::min(ms, t);
        }
        if (rc != OK) break;
        if (ci == 0) keep_ms = ms;
        if (ms < best) {
          best = ms;
          pick = c;
        }
      }
      if (best > 0.98f * keep_ms) pick = keep;
      g_fft_tuning[n][e] = rc == OK ? pick : before;
      if (out_tile) out_tile[slot] = g_fft_tuning[n][e].tile_log;
      if (out_coalesce) out_coalesce[slot] = g_fft_tuning[n][e].coalesce_bits;
    }
  }
  g_cols_aligned = aligned;
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaFreeAsync(stab, st);
  cudaFreeAsync(tab, st);
  cudaFreeAsync(src, st);
  cudaFreeAsync(buf, st);
  if (rc == ERR_CUDA) set_error(std::string("fft autotune: ") + cudaGetErrorString(cudaGetLastError()));
  return rc;
}

void get_fft_tuning(uint32_t layers, uint32_t ext, uint32_t* tile_log, uint32_t* coalesce_bits) {
  const FftTuning t = reported(g_fft_tuning[layers < 32 ? layers : 31][ext < FFT_MAX_EXT ? ext : FFT_MAX_EXT]);
  *tile_log = t.tile_log;
  *coalesce_bits = t.coalesce_bits;
}

// In-place bit reversal of one column (ColumnOps::bit_reverse_column).
__global__ void bit_reverse_kernel(uint32_t* d, uint32_t log_n) {
  uint32_t n = 1u << log_n;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t j = __brev(i) >> (32 - log_n);
    if (j > i) {
      uint32_t a = d[i];
      d[i] = d[j];
      d[j] = a;
    }
  }
}
int bit_reverse(cudaStream_t st, uint32_t* d, uint32_t log_n) {
  GS_REQUIRE(log_n <= 31, "log_n out of range");
  if (log_n == 0) return OK;
  uint32_t n = 1u << log_n;
  int blocks = (int)std::min<uint32_t>((n + 255) / 256, (uint32_t)num_sms() * 16);
  bit_reverse_kernel<<<blocks, 256, 0, st>>>(d, log_n);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}

}  // namespace gs
