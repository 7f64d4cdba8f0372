// Blake2s-256 compression for the device (RFC 7693; the reference uses the
// `blake2 = 0.10.6` crate at crates/stwo/src/core/vcs/blake2_merkle.rs:18-39).
//
// Each thread keeps the 16 message words and the 16-word working state in
// registers; the message schedule is resolved at compile time (fully unrolled
// rounds), so a compression is pure 32-bit add/xor/rotate work: IADD3 for the
// three-input adds, LOP3 for xors, PRMT/SHF for the rotations.
#pragma once
#include <cstdint>
#include "m31.cuh"

namespace gs {


constexpr uint32_t BLAKE_IV0 = 0x6A09E667u, BLAKE_IV1 = 0xBB67AE85u, BLAKE_IV2 = 0x3C6EF372u, BLAKE_IV3 = 0xA54FF53Au,
                   BLAKE_IV4 = 0x510E527Fu, BLAKE_IV5 = 0x9B05688Cu, BLAKE_IV6 = 0x1F83D9ABu, BLAKE_IV7 = 0x5BE0CD19u;
// Initial chaining value for an unkeyed 32-byte digest: IV0 ^ 0x01010020.
constexpr uint32_t BLAKE_H0 = BLAKE_IV0 ^ 0x01010020u;

GS_HD uint32_t rotr32(uint32_t x, int n) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(x, x, n);
#else
  return (x >> n) | (x << (32 - n));
#endif
}

// Rotations by 16 and 8 are byte permutes (PRMT) on the device.
GS_HD uint32_t rotr16(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __byte_perm(x, 0, 0x1032);
#else
  return rotr32(x, 16);
#endif
}
GS_HD uint32_t rotr8(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __byte_perm(x, 0, 0x0321);
#else
  return rotr32(x, 8);
#endif
}

#define GS_G(a, b, c, d, x, y)         \
  do {                                 \
    v[a] = v[a] + v[b] + (x);          \
    v[d] = rotr16(v[d] ^ v[a]);        \
    v[c] = v[c] + v[d];                \
    v[b] = rotr32(v[b] ^ v[c], 12);    \
    v[a] = v[a] + v[b] + (y);          \
    v[d] = rotr8(v[d] ^ v[a]);         \
    v[c] = v[c] + v[d];                \
    v[b] = rotr32(v[b] ^ v[c], 7);     \
  } while (0)

#define GS_ROUND(s0, s1, s2, s3, s4, s5, s6, s7, s8, s9, s10, s11, s12, s13, s14, s15) \
  do {                                                                                 \
    GS_G(0, 4, 8, 12, m[s0], m[s1]);                                                   \
    GS_G(1, 5, 9, 13, m[s2], m[s3]);                                                   \
    GS_G(2, 6, 10, 14, m[s4], m[s5]);                                                  \
    GS_G(3, 7, 11, 15, m[s6], m[s7]);                                                  \
    GS_G(0, 5, 10, 15, m[s8], m[s9]);                                                  \
    GS_G(1, 6, 11, 12, m[s10], m[s11]);                                                \
    GS_G(2, 7, 8, 13, m[s12], m[s13]);                                                 \
    GS_G(3, 4, 9, 14, m[s14], m[s15]);                                                 \
  } while (0)

// h <- compress(h, m, t, last). t = total bytes hashed so far including this block.
GS_HD void blake2s_compress(uint32_t h[8], const uint32_t m[16], uint32_t t, bool last) {
  uint32_t v[16];
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = h[i];
  v[8] = BLAKE_IV0; v[9] = BLAKE_IV1; v[10] = BLAKE_IV2; v[11] = BLAKE_IV3;
  v[12] = BLAKE_IV4 ^ t; v[13] = BLAKE_IV5; v[14] = last ? ~BLAKE_IV6 : BLAKE_IV6; v[15] = BLAKE_IV7;
  GS_ROUND(0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15);
  GS_ROUND(14, 10, 4, 8, 9, 15, 13, 6, 1, 12, 0, 2, 11, 7, 5, 3);
  GS_ROUND(11, 8, 12, 0, 5, 2, 15, 13, 10, 14, 3, 6, 7, 1, 9, 4);
  GS_ROUND(7, 9, 3, 1, 13, 12, 11, 14, 2, 6, 5, 10, 4, 0, 15, 8);
  GS_ROUND(9, 0, 5, 7, 2, 4, 10, 15, 14, 1, 11, 12, 6, 8, 3, 13);
  GS_ROUND(2, 12, 6, 10, 0, 11, 8, 3, 4, 13, 7, 5, 15, 14, 1, 9);
  GS_ROUND(12, 5, 1, 15, 14, 13, 4, 10, 0, 7, 6, 3, 9, 2, 8, 11);
  GS_ROUND(13, 11, 7, 14, 12, 1, 3, 9, 5, 0, 15, 4, 8, 6, 2, 10);
  GS_ROUND(6, 15, 14, 9, 11, 3, 0, 8, 12, 2, 13, 7, 1, 4, 10, 5);
  GS_ROUND(10, 2, 8, 4, 7, 6, 1, 5, 15, 11, 9, 14, 3, 12, 13, 0);
#pragma unroll
  for (int i = 0; i < 8; i++) h[i] ^= v[i] ^ v[i + 8];
}

#ifdef __CUDACC__
// The same compression for kernels that are bound by throughput. The xors and
// rotations (two issue cycles each on the integer ALU pipe) bound it, so no
// add goes there: a two-input add issues at full rate beside that pipe (one
// cycle), and a three-input add is an IMAD against a runtime 1 (`one`, on the
// FMA pipe) of the terms known early, then a two-input add of b, the last to
// arrive. Leaf layer of 64 x 2^20: 206 -> 196 us against one IMAD per add.
__device__ __forceinline__ uint32_t b2_imad(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
#define GS_GF(a, b, c, d, x, y)                                          \
  do {                                                                   \
    v[a] = (x < NW ? b2_imad(v[a], one, m[x]) : v[a]) + v[b];            \
    v[d] = rotr16(v[d] ^ v[a]);                                          \
    v[c] = v[c] + v[d];                                                  \
    v[b] = rotr32(v[b] ^ v[c], 12);                                      \
    v[a] = (y < NW ? b2_imad(v[a], one, m[y]) : v[a]) + v[b];            \
    v[d] = rotr8(v[d] ^ v[a]);                                           \
    v[c] = v[c] + v[d];                                                  \
    v[b] = rotr32(v[b] ^ v[c], 7);                                       \
  } while (0)
#define GS_ROUNDF(s0, s1, s2, s3, s4, s5, s6, s7, s8, s9, s10, s11, s12, s13, s14, s15) \
  do {                                                                                  \
    GS_GF(0, 4, 8, 12, s0, s1);                                                       \
    GS_GF(1, 5, 9, 13, s2, s3);                                                       \
    GS_GF(2, 6, 10, 14, s4, s5);                                                      \
    GS_GF(3, 7, 11, 15, s6, s7);                                                      \
    GS_GF(0, 5, 10, 15, s8, s9);                                                      \
    GS_GF(1, 6, 11, 12, s10, s11);                                                    \
    GS_GF(2, 7, 8, 13, s12, s13);                                                     \
    GS_GF(3, 4, 9, 14, s14, s15);                                                     \
  } while (0)
// NW: message words that can be nonzero, the first ones.
template <int NW = 16>
__device__ __forceinline__ void blake2s_compress_f(uint32_t h[8], const uint32_t m[16], uint32_t t, bool last,
                                                   uint32_t one) {
  uint32_t v[16];
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = h[i];
  v[8] = BLAKE_IV0; v[9] = BLAKE_IV1; v[10] = BLAKE_IV2; v[11] = BLAKE_IV3;
  v[12] = BLAKE_IV4 ^ t; v[13] = BLAKE_IV5; v[14] = last ? ~BLAKE_IV6 : BLAKE_IV6; v[15] = BLAKE_IV7;
  GS_ROUNDF(0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15);
  GS_ROUNDF(14, 10, 4, 8, 9, 15, 13, 6, 1, 12, 0, 2, 11, 7, 5, 3);
  GS_ROUNDF(11, 8, 12, 0, 5, 2, 15, 13, 10, 14, 3, 6, 7, 1, 9, 4);
  GS_ROUNDF(7, 9, 3, 1, 13, 12, 11, 14, 2, 6, 5, 10, 4, 0, 15, 8);
  GS_ROUNDF(9, 0, 5, 7, 2, 4, 10, 15, 14, 1, 11, 12, 6, 8, 3, 13);
  GS_ROUNDF(2, 12, 6, 10, 0, 11, 8, 3, 4, 13, 7, 5, 15, 14, 1, 9);
  GS_ROUNDF(12, 5, 1, 15, 14, 13, 4, 10, 0, 7, 6, 3, 9, 2, 8, 11);
  GS_ROUNDF(13, 11, 7, 14, 12, 1, 3, 9, 5, 0, 15, 4, 8, 6, 2, 10);
  GS_ROUNDF(6, 15, 14, 9, 11, 3, 0, 8, 12, 2, 13, 7, 1, 4, 10, 5);
  GS_ROUNDF(10, 2, 8, 4, 7, 6, 1, 5, 15, 11, 9, 14, 3, 12, 13, 0);
#pragma unroll
  for (int i = 0; i < 8; i++) h[i] ^= v[i] ^ v[i + 8];
}
#endif

#ifdef __CUDACC__
// One compression of a single-block message by four lanes, for levels with so
// few nodes that a lone warp's latency is all that counts: lane j = threadIdx.x
// & 3 holds column j of the state, so a G step is one chain per lane, not four
// that queue for the ALU pipe, and a diagonal step is the same G on a, c and d
// from the neighbouring lanes (b, the last word a G writes and the first the
// next one reads, stays where it is, so the shuffles run beside the G's tail).
// The message is read from shared memory word by word: each round's four byte
// offsets of a lane are packed in one word, and a dot product with 1 << 8k
// adds byte k to the message's address. 1386 cycles against 1690 for one lane.
__host__ __device__ constexpr uint32_t blake2s_sigma(int r, int k) {
  constexpr uint8_t S[10][16] = {
      {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15}, {14, 10, 4, 8, 9, 15, 13, 6, 1, 12, 0, 2, 11, 7, 5, 3},
      {11, 8, 12, 0, 5, 2, 15, 13, 10, 14, 3, 6, 7, 1, 9, 4}, {7, 9, 3, 1, 13, 12, 11, 14, 2, 6, 5, 10, 4, 0, 15, 8},
      {9, 0, 5, 7, 2, 4, 10, 15, 14, 1, 11, 12, 6, 8, 3, 13}, {2, 12, 6, 10, 0, 11, 8, 3, 4, 13, 7, 5, 15, 14, 1, 9},
      {12, 5, 1, 15, 14, 13, 4, 10, 0, 7, 6, 3, 9, 2, 8, 11}, {13, 11, 7, 14, 12, 1, 3, 9, 5, 0, 15, 4, 8, 6, 2, 10},
      {6, 15, 14, 9, 11, 3, 0, 8, 12, 2, 13, 7, 1, 4, 10, 5}, {10, 2, 8, 4, 7, 6, 1, 5, 15, 11, 9, 14, 3, 12, 13, 0}};
  return S[r][k];
}
// Lane j's byte offsets in round r: column words 2j, 2j + 1, then those of the
// diagonal whose b is b_j, diagonal (j + 3) mod 4.
__host__ __device__ constexpr uint32_t blake2s_quad_offsets(int r, int j) {
  const int g = (j + 3) & 3;
  return 4u * (blake2s_sigma(r, 2 * j) | blake2s_sigma(r, 2 * j + 1) << 8 | blake2s_sigma(r, 8 + 2 * g) << 16 |
               blake2s_sigma(r, 9 + 2 * g) << 24);
}
// The offsets in shared memory, [round][lane]: filled by threads 0..3 (the
// selects of constants cost a tenth of a compression when done in it).
__device__ __forceinline__ void blake2s_quad_table(uint32_t tab[40]) {
  const uint32_t j = threadIdx.x;
  if (j >= 4) return;
#define GS_QUAD_ROW(r)                                                                                            \
  do {                                                                                                            \
    constexpr uint32_t o0 = blake2s_quad_offsets(r, 0), o1 = blake2s_quad_offsets(r, 1),                          \
                       o2 = blake2s_quad_offsets(r, 2), o3 = blake2s_quad_offsets(r, 3);                          \
    tab[4 * r + j] = j & 2u ? (j & 1u ? o3 : o2) : (j & 1u ? o1 : o0);                                            \
  } while (0)
  GS_QUAD_ROW(0); GS_QUAD_ROW(1); GS_QUAD_ROW(2); GS_QUAD_ROW(3); GS_QUAD_ROW(4);
  GS_QUAD_ROW(5); GS_QUAD_ROW(6); GS_QUAD_ROW(7); GS_QUAD_ROW(8); GS_QUAD_ROW(9);
#undef GS_QUAD_ROW
}
// h0, h1: words j and 4 + j of the hash. All 32 lanes take part; a barrier lies
// between the stores of the message (and the table) by other lanes and this.
__device__ __forceinline__ void blake2s_quad(const uint32_t* tab, const uint4* msg, uint32_t bytes, uint32_t& h0,
                                             uint32_t& h1) {
  const uint32_t j = threadIdx.x & 3u;
  auto by_lane = [&](uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3) {
    return j & 2u ? (j & 1u ? x3 : x2) : (j & 1u ? x1 : x0);
  };
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(msg);
  auto fetch = [&](uint32_t offsets, uint32_t w[4]) {
    uint32_t at[4];
#pragma unroll
    for (int k = 0; k < 4; k++) at[k] = __dp4a(offsets, 1u << (8 * k), base);
#pragma unroll
    for (int k = 0; k < 4; k++) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[k]) : "r"(at[k]) : "memory");
  };
  uint32_t m[4], next[4];
  fetch(tab[j], m);
  uint32_t off = tab[4 + j];
  const uint32_t ia = by_lane(BLAKE_H0, BLAKE_IV1, BLAKE_IV2, BLAKE_IV3);
  const uint32_t ib = by_lane(BLAKE_IV4, BLAKE_IV5, BLAKE_IV6, BLAKE_IV7);
  uint32_t a = ia, b = ib, c = by_lane(BLAKE_IV0, BLAKE_IV1, BLAKE_IV2, BLAKE_IV3);
  uint32_t d = by_lane(BLAKE_IV4 ^ bytes, BLAKE_IV5, ~BLAKE_IV6, BLAKE_IV7);
  const int up = (j + 1) & 3, across = (j + 2) & 3, down = (j + 3) & 3;
  auto g = [&](uint32_t x, uint32_t y) {
    a = a + b + x;
    d = rotr16(d ^ a);
    c = c + d;
    b = rotr32(b ^ c, 12);
    a = a + b + y;
    d = rotr8(d ^ a);
    c = c + d;
    b = rotr32(b ^ c, 7);
  };
#pragma unroll
  for (int r = 0; r < 10; r++) {
    if (r < 9) fetch(off, next);
    if (r < 8) off = tab[4 * (r + 2) + j];
    g(m[0], m[1]);
    a = __shfl_sync(0xffffffffu, a, down, 4);
    d = __shfl_sync(0xffffffffu, d, across, 4);
    c = __shfl_sync(0xffffffffu, c, up, 4);
    g(m[2], m[3]);
    a = __shfl_sync(0xffffffffu, a, up, 4);
    d = __shfl_sync(0xffffffffu, d, across, 4);
    c = __shfl_sync(0xffffffffu, c, down, 4);
#pragma unroll
    for (int k = 0; k < 4; k++) m[k] = next[k];
  }
  h0 = ia ^ a ^ c;
  h1 = ib ^ b ^ d;
}
#endif

GS_HD void blake2s_init(uint32_t h[8]) {
  h[0] = BLAKE_H0; h[1] = BLAKE_IV1; h[2] = BLAKE_IV2; h[3] = BLAKE_IV3;
  h[4] = BLAKE_IV4; h[5] = BLAKE_IV5; h[6] = BLAKE_IV6; h[7] = BLAKE_IV7;
}

}  // namespace gs
