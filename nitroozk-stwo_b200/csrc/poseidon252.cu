// Poseidon252 Merkle hashing on the device: MerkleOps<Poseidon252MerkleHasher>
// ::commit_on_layer (crates/stwo/src/core/vcs/poseidon252_merkle.rs:18-72;
// reference CUDA poseidon252_commit_on_first_layer / _with_previous,
// stwo_cuda/bindings.rs:592-612).
//
// The hash is Starknet's Poseidon (the Hades permutation of the crate
// starknet-crypto 0.6.2 that the reference calls): field p = 2^251 +
// 17·2^192 + 1, state of 3 elements, x^3 S-box, 4 full + 83 partial + 4 full
// rounds, MDS [[3, 1, 1], [1, -1, 1], [1, 1, -2]], round constants from
// poseidon252_constants.py.
//
//   hash_node(children, values): poseidon_hash(l, r) when there are children
//   and no values; otherwise poseidon_hash_many([l, r,] felts of the values,
//   8 M31 values per felt shifted in 31 bits at a time, a shorter last word
//   carrying its length at bit 248).
//
// Field elements live in registers as 8 little-endian 32-bit limbs in
// Montgomery form (R = 2^256). The modulus is sparse, limbs [1, 0, 0, 0, 0, 0,
// 17, 2^27], and p = 1 mod 2^192, so 192 bits of a product reduce in one step
// of shifts and a subtraction. Hashes in memory are the reference's device
// layout: 32 bytes, big-endian.
#include "runtime.cuh"
#include <cstring>

namespace gs {

struct Felt {
  uint32_t v[8];
};

#include "poseidon252_constants.inc"

// Carry chains in PTX (add.cc / addc, mad.lo.cc / madc.hi.cc): one
// instruction per limb, the carry in the flag.

// t -> t - p when t >= p (t < 2p); branch-free select
__device__ __forceinline__ void reduce_once(uint32_t t[8]) {
  uint32_t d[8], bw;
  asm("sub.cc.u32 %0, %9, 1;\n\t"
      "subc.cc.u32 %1, %10, 0;\n\t"
      "subc.cc.u32 %2, %11, 0;\n\t"
      "subc.cc.u32 %3, %12, 0;\n\t"
      "subc.cc.u32 %4, %13, 0;\n\t"
      "subc.cc.u32 %5, %14, 0;\n\t"
      "subc.cc.u32 %6, %15, 17;\n\t"
      "subc.cc.u32 %7, %16, 0x08000000;\n\t"
      "subc.u32 %8, 0, 0;"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(bw)
      : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]));
#pragma unroll
  for (int j = 0; j < 8; j++) t[j] = (t[j] & bw) | (d[j] & ~bw);  // borrow: t < p, keep it
}

// Products. p = 1 + q·2^192 with q = 2^59 + 17, so the Montgomery reduction
// needs no product by p: T - x·p with x = the low 192 bits of T is divisible
// by 2^192 and leaves (T >> 192) - x·q, a shift by 4 added to x, a shift by
// 59, and one subtraction; a second step takes 64 bits the same way. So a
// product is a plain 512-bit product, then one lump reduction by R = 2^256.
//
// The 512-bit product runs in rows over two accumulators, one for the
// products that land on even 32-bit columns (E) and one for odd columns (O):
// neighbouring products of a row then fill separate 64-bit columns, and each
// is one wide multiply-add with the carry of its row (mad.lo.cc / madc.hi.cc
// on one column pair): 64 wide multiplies instead of 64 low and 64 high ones,
// which cost 4 against 2 + 4 issue cycles per warp. A square takes 28 + 8.
//
// The subtractions can leave a negative value, so a multiple of p is added to
// T: k·p·2^256 + p·2^192 (its limbs enter as the starting values of the
// accumulators' fresh columns, at no instruction). The result is then at
// least (k - 1)·p and below T / 2^256 + (k + 1/1000)·p.
//
// Measured against a limb-by-limb reduction (CIOS, low and high multiplies):
// 97 k -> 37.7 k warp instructions per permutation, so a lone warp, which a
// small tree level is, takes 105 -> 60 us (it now waits on the carry chains:
// 3.1 cycles per instruction, the multiplier busy for half of them), and a
// Wide-Fibonacci 2^16 x 100 proof over this hash 30.5 -> 16.1 ms.

// Columns t[0..2n) += (a0, a1, ...) · b, one wide multiply-add per pair of
// columns; in the c forms the carry of the last goes to `top` (= top0 + carry).
__device__ __forceinline__ void wchain1c(uint32_t* t, uint32_t a0, uint32_t b, uint32_t& top, uint32_t top0) {
  asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
      "addc.u32 %2, %5, 0;"
      : "+r"(t[0]), "+r"(t[1]), "=r"(top)
      : "r"(a0), "r"(b), "r"(top0));
}
__device__ __forceinline__ void wchain1(uint32_t* t, uint32_t a0, uint32_t b) {
  asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\t"
      "madc.hi.u32 %1, %2, %3, %1;"
      : "+r"(t[0]), "+r"(t[1])
      : "r"(a0), "r"(b));
}
__device__ __forceinline__ void wchain2c(uint32_t* t, uint32_t a0, uint32_t a1, uint32_t b, uint32_t& top, uint32_t top0) {
  asm("mad.lo.cc.u32 %0, %5, %7, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
      "addc.u32 %4, %8, 0;"
      : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "=r"(top)
      : "r"(a0), "r"(a1), "r"(b), "r"(top0));
}
__device__ __forceinline__ void wchain2(uint32_t* t, uint32_t a0, uint32_t a1, uint32_t b) {
  asm("mad.lo.cc.u32 %0, %4, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
      "madc.hi.u32 %3, %5, %6, %3;"
      : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3])
      : "r"(a0), "r"(a1), "r"(b));
}
__device__ __forceinline__ void wchain3c(uint32_t* t, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t b, uint32_t& top, uint32_t top0) {
  asm("mad.lo.cc.u32 %0, %7, %10, %0;\n\t"
      "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
      "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
      "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
      "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
      "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
      "addc.u32 %6, %11, 0;"
      : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "=r"(top)
      : "r"(a0), "r"(a1), "r"(a2), "r"(b), "r"(top0));
}
__device__ __forceinline__ void wchain3(uint32_t* t, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t b) {
  asm("mad.lo.cc.u32 %0, %6, %9, %0;\n\t"
      "madc.hi.cc.u32 %1, %6, %9, %1;\n\t"
      "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
      "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
      "madc.lo.cc.u32 %4, %8, %9, %4;\n\t"
      "madc.hi.u32 %5, %8, %9, %5;"
      : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5])
      : "r"(a0), "r"(a1), "r"(a2), "r"(b));
}
__device__ __forceinline__ void wchain4c(uint32_t* t, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b, uint32_t& top, uint32_t top0) {
  asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\t"
      "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
      "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
      "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
      "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
      "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
      "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
      "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
      "addc.u32 %8, %14, 0;"
      : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]), "=r"(top)
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b), "r"(top0));
}
__device__ __forceinline__ void wchain4(uint32_t* t, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b) {
  asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\t"
      "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
      "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
      "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
      "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
      "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
      "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
      "madc.hi.u32 %7, %11, %12, %7;"
      : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b));
}

// the same over the eight squares, no carry out
__device__ __forceinline__ void sqchain8(uint32_t t[16], const Felt& a) {
  asm("mad.lo.cc.u32 %0, %16, %16, %0;\n\t"
      "madc.hi.cc.u32 %1, %16, %16, %1;\n\t"
      "madc.lo.cc.u32 %2, %17, %17, %2;\n\t"
      "madc.hi.cc.u32 %3, %17, %17, %3;\n\t"
      "madc.lo.cc.u32 %4, %18, %18, %4;\n\t"
      "madc.hi.cc.u32 %5, %18, %18, %5;\n\t"
      "madc.lo.cc.u32 %6, %19, %19, %6;\n\t"
      "madc.hi.cc.u32 %7, %19, %19, %7;\n\t"
      "madc.lo.cc.u32 %8, %20, %20, %8;\n\t"
      "madc.hi.cc.u32 %9, %20, %20, %9;\n\t"
      "madc.lo.cc.u32 %10, %21, %21, %10;\n\t"
      "madc.hi.cc.u32 %11, %21, %21, %11;\n\t"
      "madc.lo.cc.u32 %12, %22, %22, %12;\n\t"
      "madc.hi.cc.u32 %13, %22, %22, %13;\n\t"
      "madc.lo.cc.u32 %14, %23, %23, %14;\n\t"
      "madc.hi.u32 %15, %23, %23, %15;"
      : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]), "+r"(t[8]),
        "+r"(t[9]), "+r"(t[10]), "+r"(t[11]), "+r"(t[12]), "+r"(t[13]), "+r"(t[14]), "+r"(t[15])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]));
}
// T[j] = e[j] + o[j - 1], columns 1..15
__device__ __forceinline__ void add_columns(uint32_t T[16], const uint32_t e[16], const uint32_t o[16]) {
  asm("add.cc.u32 %0, %15, %30;\n\t"
      "addc.cc.u32 %1, %16, %31;\n\t"
      "addc.cc.u32 %2, %17, %32;\n\t"
      "addc.cc.u32 %3, %18, %33;\n\t"
      "addc.cc.u32 %4, %19, %34;\n\t"
      "addc.cc.u32 %5, %20, %35;\n\t"
      "addc.cc.u32 %6, %21, %36;\n\t"
      "addc.cc.u32 %7, %22, %37;\n\t"
      "addc.cc.u32 %8, %23, %38;\n\t"
      "addc.cc.u32 %9, %24, %39;\n\t"
      "addc.cc.u32 %10, %25, %40;\n\t"
      "addc.cc.u32 %11, %26, %41;\n\t"
      "addc.cc.u32 %12, %27, %42;\n\t"
      "addc.cc.u32 %13, %28, %43;\n\t"
      "addc.u32 %14, %29, %44;"
      : "=&r"(T[1]), "=&r"(T[2]), "=&r"(T[3]), "=&r"(T[4]), "=&r"(T[5]), "=&r"(T[6]), "=&r"(T[7]), "=&r"(T[8]),
        "=&r"(T[9]), "=&r"(T[10]), "=&r"(T[11]), "=&r"(T[12]), "=&r"(T[13]), "=&r"(T[14]), "=&r"(T[15])
      : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]), "r"(e[10]),
        "r"(e[11]), "r"(e[12]), "r"(e[13]), "r"(e[14]), "r"(e[15]), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]),
        "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]), "r"(o[12]),
        "r"(o[13]), "r"(o[14]));
}

// T = a·b + (k·p·2^64 + p)·2^192. a, b < 2^255 with a·b < 2^510.
__device__ __forceinline__ void mul_wide8(uint32_t K, const Felt& a, const Felt& b, uint32_t T[16]) {
  uint32_t e[16], o[16];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint64_t pe = (uint64_t)a.v[2 * j] * b.v[0] + (j == 3 ? 1u : 0u);  // column 6: + 1
    const uint64_t po = (uint64_t)a.v[2 * j + 1] * b.v[0];
    e[2 * j] = (uint32_t)pe;
    e[2 * j + 1] = (uint32_t)(pe >> 32);
    o[2 * j] = (uint32_t)po;
    o[2 * j + 1] = (uint32_t)(po >> 32);
  }
  e[8] = K;
#pragma unroll
  for (int i = 1; i < 8; i++) {
    // odd rows put their even-limb products on odd columns
    uint32_t* x = i & 1 ? o : e;
    uint32_t* y = i & 1 ? e : o;
    const int xb = i & 1 ? i - 1 : i, yb = i & 1 ? i + 1 : i;
    wchain4c(x + xb, a.v[0], a.v[2], a.v[4], a.v[6], b.v[i], x[xb + 8], i == 4 ? 17u : i == 6 ? 17u * K : 0u);
    y[yb + 7] = i == 5 ? 0x08000000u : i == 7 ? K << 27 : 0u;
    wchain4(y + yb, a.v[1], a.v[3], a.v[5], a.v[7], b.v[i]);
  }
  T[0] = e[0];
  add_columns(T, e, o);
}

// T = a^2 + 2·(p·2^64 + p)·2^192, a < 2^255. Cross products once, doubled,
// then the squares in one chain.
__device__ __forceinline__ void sqr_wide8(const Felt& a, uint32_t T[16]) {
  uint32_t e[16], o[16], c[16];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint64_t po = (uint64_t)a.v[0] * a.v[2 * j + 1];
    o[2 * j] = (uint32_t)po;
    o[2 * j + 1] = (uint32_t)(po >> 32);
  }
#pragma unroll
  for (int j = 1; j < 4; j++) {
    const uint64_t pe = (uint64_t)a.v[0] * a.v[2 * j] + (j == 3 ? 1u : 0u);  // column 6: + 1
    e[2 * j] = (uint32_t)pe;
    e[2 * j + 1] = (uint32_t)(pe >> 32);
  }
  e[0] = e[1] = 0;
  e[8] = 1;
  e[9] = 0;
  wchain3c(o + 2, a.v[2], a.v[4], a.v[6], a.v[1], o[8], 0);
  wchain3(e + 4, a.v[3], a.v[5], a.v[7], a.v[1]);
  o[9] = 0;
  wchain3(o + 4, a.v[3], a.v[5], a.v[7], a.v[2]);
  wchain2c(e + 6, a.v[4], a.v[6], a.v[2], e[10], 0);
  wchain2c(o + 6, a.v[4], a.v[6], a.v[3], o[10], 0);
  e[11] = 0;
  wchain2(e + 8, a.v[5], a.v[7], a.v[3]);
  o[11] = 0;
  wchain2(o + 8, a.v[5], a.v[7], a.v[4]);
  wchain1c(e + 10, a.v[6], a.v[4], e[12], 17u);
  wchain1c(o + 10, a.v[6], a.v[5], o[12], 0);
  e[13] = 0x08000000u;
  wchain1(e + 12, a.v[7], a.v[5]);
  o[13] = 0;
  wchain1(o + 12, a.v[7], a.v[6]);
  o[14] = 0;
  e[14] = 17u;
  e[15] = 0x08000000u;
  c[0] = 0;
  add_columns(c, e, o);
  T[0] = 0;
#pragma unroll
  for (int j = 15; j >= 1; j--) T[j] = __funnelshift_l(c[j - 1], c[j], 1);
  sqchain8(T, a);
}

// (T / 2^256) mod p for T = product + k·p·2^256 + p·2^192, in two steps of 192
// and 64 bits: T - x·p with x the low bits, x·(2^59 + 17) from shifts.
__device__ __forceinline__ Felt redc(const uint32_t T[16]) {
  uint32_t s[8], z[8], r[10];
  s[0] = T[0] << 4;
  z[0] = T[0] << 27;
#pragma unroll
  for (int j = 1; j < 6; j++) {
    s[j] = __funnelshift_l(T[j - 1], T[j], 4);
    z[j] = __funnelshift_l(T[j - 1], T[j], 27);
  }
  s[6] = T[5] >> 28;
  z[6] = T[5] >> 5;
  // s = 16 x + x, then + x·2^59 (limbs 1..7)
  asm("add.cc.u32 %0, %0, %7;\n\t"
      "addc.cc.u32 %1, %1, %8;\n\t"
      "addc.cc.u32 %2, %2, %9;\n\t"
      "addc.cc.u32 %3, %3, %10;\n\t"
      "addc.cc.u32 %4, %4, %11;\n\t"
      "addc.cc.u32 %5, %5, %12;\n\t"
      "addc.u32 %6, %6, 0;"
      : "+r"(s[0]), "+r"(s[1]), "+r"(s[2]), "+r"(s[3]), "+r"(s[4]), "+r"(s[5]), "+r"(s[6])
      : "r"(T[0]), "r"(T[1]), "r"(T[2]), "r"(T[3]), "r"(T[4]), "r"(T[5]));
  asm("add.cc.u32 %0, %0, %7;\n\t"
      "addc.cc.u32 %1, %1, %8;\n\t"
      "addc.cc.u32 %2, %2, %9;\n\t"
      "addc.cc.u32 %3, %3, %10;\n\t"
      "addc.cc.u32 %4, %4, %11;\n\t"
      "addc.cc.u32 %5, %5, %12;\n\t"
      "addc.u32 %6, %13, 0;"
      : "+r"(s[1]), "+r"(s[2]), "+r"(s[3]), "+r"(s[4]), "+r"(s[5]), "+r"(s[6]), "=r"(s[7])
      : "r"(z[0]), "r"(z[1]), "r"(z[2]), "r"(z[3]), "r"(z[4]), "r"(z[5]), "r"(z[6]));
  asm("sub.cc.u32 %0, %10, %20;\n\t"
      "subc.cc.u32 %1, %11, %21;\n\t"
      "subc.cc.u32 %2, %12, %22;\n\t"
      "subc.cc.u32 %3, %13, %23;\n\t"
      "subc.cc.u32 %4, %14, %24;\n\t"
      "subc.cc.u32 %5, %15, %25;\n\t"
      "subc.cc.u32 %6, %16, %26;\n\t"
      "subc.cc.u32 %7, %17, %27;\n\t"
      "subc.cc.u32 %8, %18, 0;\n\t"
      "subc.u32 %9, %19, 0;"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]),
        "=&r"(r[8]), "=&r"(r[9])
      : "r"(T[6]), "r"(T[7]), "r"(T[8]), "r"(T[9]), "r"(T[10]), "r"(T[11]), "r"(T[12]), "r"(T[13]), "r"(T[14]),
        "r"(T[15]), "r"(s[0]), "r"(s[1]), "r"(s[2]), "r"(s[3]), "r"(s[4]), "r"(s[5]), "r"(s[6]), "r"(s[7]));
  // 64 bits more: y = r[0..1], y·q lands on limbs 6..9
  uint32_t w0 = r[0] << 4, w1 = __funnelshift_l(r[0], r[1], 4), w2 = r[1] >> 28, w3;
  asm("add.cc.u32 %0, %0, %3;\n\t"
      "addc.cc.u32 %1, %1, %4;\n\t"
      "addc.u32 %2, %2, 0;"
      : "+r"(w0), "+r"(w1), "+r"(w2)
      : "r"(r[0]), "r"(r[1]));
  asm("add.cc.u32 %0, %0, %3;\n\t"
      "addc.cc.u32 %1, %1, %4;\n\t"
      "addc.u32 %2, %5, 0;"
      : "+r"(w1), "+r"(w2), "=r"(w3)
      : "r"(r[0] << 27), "r"(__funnelshift_l(r[0], r[1], 27)), "r"(r[1] >> 5));
  Felt f;
#pragma unroll
  for (int j = 0; j < 4; j++) f.v[j] = r[2 + j];
  asm("sub.cc.u32 %0, %4, %8;\n\t"
      "subc.cc.u32 %1, %5, %9;\n\t"
      "subc.cc.u32 %2, %6, %10;\n\t"
      "subc.u32 %3, %7, %11;"
      : "=&r"(f.v[4]), "=&r"(f.v[5]), "=&r"(f.v[6]), "=&r"(f.v[7])
      : "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(w0), "r"(w1), "r"(w2), "r"(w3));
  return f;
}

// a·b / 2^256 mod p: at least (K - 1)·p, below a·b / 2^256 + (K + 1/1000)·p.
// The top limb of a stays below 2^31.
__device__ __forceinline__ Felt fmul_k(uint32_t K, const Felt& a, const Felt& b) {
  uint32_t T[16];
  mul_wide8(K, a, b, T);
  return redc(T);
}
// Below p, for a·b < 0.9·2^256·p (the product is then below 2p).
__device__ __forceinline__ Felt fmul(const Felt& a, const Felt& b) {
  Felt r = fmul_k(1, a, b);
  reduce_once(r.v);
  return r;
}
// x^3: at least (K - 1)·p. For x <= 11p (below 2^254.5) the square is below
// (121/32 + 2 + 1/1000)·p < 5.8p and the cube below (5.8·11/32 + K)·p < (K + 2)·p.
__device__ __forceinline__ Felt fcube(uint32_t K, const Felt& x) {
  uint32_t T[16];
  sqr_wide8(x, T);
  return fmul_k(K, x, redc(T));
}


// a + b without reduction (callers keep the sum below 2^256)
__device__ __forceinline__ Felt ladd(const Felt& a, const Felt& b) {
  Felt r;
  asm("add.cc.u32 %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32 %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
        "=r"(r.v[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  return r;
}
// a - b without reduction (callers guarantee a >= b)
__device__ __forceinline__ Felt lsub(const Felt& a, const Felt& b) {
  Felt r;
  asm("sub.cc.u32 %0, %8, %16;\n\t"
      "subc.cc.u32 %1, %9, %17;\n\t"
      "subc.cc.u32 %2, %10, %18;\n\t"
      "subc.cc.u32 %3, %11, %19;\n\t"
      "subc.cc.u32 %4, %12, %20;\n\t"
      "subc.cc.u32 %5, %13, %21;\n\t"
      "subc.cc.u32 %6, %14, %22;\n\t"
      "subc.u32 %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
        "=r"(r.v[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  return r;
}
// x < 2^255 -> below 2p: with q = x >> 251, x - max(q - 1, 0)·p lies in
// [p - q·(17·2^192 + 1), 2^251 + p) when q > 0 (and is x < 2^251 when q = 0):
// no compare, no select.
__device__ __forceinline__ Felt lreduce(const Felt& x) {
  const uint32_t q = x.v[7] >> 27;
  const uint32_t k = q > 0 ? q - 1 : 0;
  Felt r;
  asm("sub.cc.u32 %0, %8, %16;\n\t"
      "subc.cc.u32 %1, %9, 0;\n\t"
      "subc.cc.u32 %2, %10, 0;\n\t"
      "subc.cc.u32 %3, %11, 0;\n\t"
      "subc.cc.u32 %4, %12, 0;\n\t"
      "subc.cc.u32 %5, %13, 0;\n\t"
      "subc.cc.u32 %6, %14, %17;\n\t"
      "subc.u32 %7, %15, %18;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
        "=r"(r.v[7])
      : "r"(x.v[0]), "r"(x.v[1]), "r"(x.v[2]), "r"(x.v[3]), "r"(x.v[4]), "r"(x.v[5]), "r"(x.v[6]), "r"(x.v[7]),
        "r"(k), "r"(k * 17u), "r"(k << 27));
  return r;
}

__device__ __forceinline__ Felt fadd(const Felt& a, const Felt& b) {
  uint32_t t[8];
  asm("add.cc.u32 %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32 %7, %15, %23;"
      : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  reduce_once(t);  // a + b < 2p < 2^253
  Felt r;
#pragma unroll
  for (int j = 0; j < 8; j++) r.v[j] = t[j];
  return r;
}

// MDS [[3, 1, 1], [1, -1, 1], [1, 1, -2]] on s0, s1 < 2p and 2p <= s2 < 5p (a
// cube with K = 3): s0 + s2 - s1 is non-negative as it stands, and
// s0 + s1 - 2 s2 is with the 10p that `c` carries besides the next round's
// constant for s2. s0 and s1 come back below 2p; s2 is left at most
// 2p + 2p + 11p - 4p = 11p, which the next cube accepts.
__device__ __forceinline__ void mds(Felt s[3], const Felt& c) {
  const Felt u = ladd(s[0], s[2]), w = ladd(s[0], s[1]);
  const Felt a0 = ladd(ladd(u, w), s[0]);
  const Felt a1 = lsub(u, s[1]);
  const Felt a2 = lsub(lsub(ladd(w, c), s[2]), s[2]);
  s[0] = lreduce(a0);
  s[1] = lreduce(a1);
  s[2] = a2;
}

// The permutation with compressed partial rounds (one constant each, added
// to s2; the folded remainder sits in the first of the last 4 full rounds'
// constants): the same permutation, two constant additions fewer per
// partial round (poseidon252_constants.py derives and checks the form). The
// constant of s2 is added by the MDS before its round.
// Bounds: the state comes in below 3.5p (below 2p, or after absorbing a
// block), s0 and s1 enter every cube below 4.5p and s2 below 11p.
__device__ __forceinline__ void hades(Felt s[3]) {
  s[2] = ladd(s[2], P252_FULL_RC[2]);
#pragma unroll 1
  for (int half = 0; half < 2; half++) {
#pragma unroll 1
    for (int r = 0; r < 4; r++) {
#pragma unroll
      for (int j = 0; j < 2; j++) s[j] = fcube(1, ladd(s[j], P252_FULL_RC[3 * (4 * half + r) + j]));
      s[2] = fcube(3, s[2]);
      mds(s, P252_S2_NEXT[half ? 87 + r : r]);
    }
    if (half == 0)
#pragma unroll 1
      for (int k = 0; k < 83; k++) {
        s[2] = fcube(3, s[2]);
        mds(s, P252_S2_NEXT[4 + k]);
      }
  }
  s[2] = lreduce(s[2]);
}

// 32 big-endian bytes (as 8 little-endian-stored words) <-> canonical limbs
__device__ __forceinline__ Felt from_be_words(const uint32_t w[8]) {
  Felt x;
#pragma unroll
  for (int k = 0; k < 8; k++) x.v[7 - k] = __byte_perm(w[k], 0, 0x0123);
  return x;
}
__device__ __forceinline__ void to_be_words(const Felt& x, uint32_t w[8]) {
#pragma unroll
  for (int k = 0; k < 8; k++) w[k] = __byte_perm(x.v[7 - k], 0, 0x0123);
}
// any 256-bit x, to below 2p (below 1.1p for x < p)
__device__ __forceinline__ Felt to_mont(const Felt& x) { return fmul_k(1, P252_R2, x); }
__device__ __forceinline__ Felt from_mont(const Felt& x) {
  Felt one{};
  one.v[0] = 1;
  return fmul(x, one);
}

__device__ __forceinline__ Felt load_hash(const uint8_t* base, size_t i) {
  const uint4* p = reinterpret_cast<const uint4*>(base + 32 * i);
  const uint4 a = __ldg(p), b = __ldg(p + 1);
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  return to_mont(from_be_words(w));
}
__device__ __forceinline__ void store_hash(uint8_t* base, size_t i, const Felt& m) {
  uint32_t w[8];
  to_be_words(from_mont(m), w);
  uint4* p = reinterpret_cast<uint4*>(base + 32 * i);
  p[0] = make_uint4(w[0], w[1], w[2], w[3]);
  p[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// Value k of a node's input sequence: the children (when there is a previous
// layer), then the column words of 8 values each.
__device__ __forceinline__ Felt node_value(uint32_t k, size_t i, const uint8_t* prev,
                                           const Cols& cols, uint32_t n_cols) {
  if (prev) {
    if (k < 2) return load_hash(prev, 2 * i + k);
    k -= 2;
  }
  const uint32_t c0 = 8 * k;
  const uint32_t len = n_cols - c0 < 8 ? n_cols - c0 : 8;
  Felt f{};
  for (uint32_t q = 0; q < len; q++) {
    const uint32_t v = __ldg(cols[c0 + q] + i);
    // f = f << 31 | v
#pragma unroll
    for (int j = 7; j >= 1; j--) f.v[j] = (f.v[j] << 31) | (f.v[j - 1] >> 1);
    f.v[0] = (f.v[0] << 31) | v;
  }
  if (len < 8) f.v[7] += len << 24;  // length at bit 248
  return to_mont(f);
}

// One node per thread: children from `prev` (or none) and columns [0, n_cols).
// poseidon_hash_many of m values absorbs blocks of two from the sequence
// values, 1, 0: m / 2 + 1 permutations; poseidon_hash(l, r) (children and no
// columns) is one permutation of (l, r, 2). Either way one call site of the
// permutation, inlined with the state in registers.
__global__ void __launch_bounds__(128) poseidon252_layer_kernel(uint32_t log_size, const uint8_t* __restrict__ prev,
                                                                Cols cols, uint32_t n_cols,
                                                                uint8_t* __restrict__ out) {
  after_previous(prev, cols);
  const size_t n = (size_t)1 << log_size;
  const bool node_only = prev && n_cols == 0;
  const uint32_t m = (prev ? 2u : 0u) + (n_cols + 7) / 8;  // values
  const uint32_t n_blocks = node_only ? 1u : m / 2 + 1;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    Felt s[3] = {};
    if (node_only) s[2] = P252_TWO;
    for (uint32_t b = 0; b < n_blocks; b++) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint32_t k = 2 * b + h;
        if (k < m) s[h] = ladd(s[h], node_value(k, i, prev, cols, n_cols));
        else if (k == m && !node_only) s[h] = ladd(s[h], P252_ONE);
      }
      hades(s);
    }
    store_hash(out, i, s[0]);
  }
}

// Node levels with few nodes, where one permutation's latency is the whole
// time: a block of three warps takes 32 nodes, lane i node i, and in a full
// round warp w cubes state element w, so a full round costs one cube and an
// exchange through shared memory instead of three cubes. In a partial round
// only s2 is cubed: warp 0 does that and nothing else, while warp 1 updates s0
// and s1 with the cube of the round before and hands back s0 + s1 + constant,
// which warp 0 picks up between its square and its product. With at most 32 nodes the block goes on to the root, the hashes of a level
// handed to the next in Montgomery form. One level: 60 -> 39 us
// (two cubes fewer to wait for in each full round, the rest the additions).
struct Levels252 {
  uint8_t* p[6];  // level L: 2^L hashes
};
__global__ void __launch_bounds__(96) poseidon252_trio_kernel(uint32_t log_size, const uint8_t* __restrict__ prev,
                                                              uint8_t* out, Levels252 up, uint32_t to_root) {
  after_previous(prev);
  __shared__ uint32_t ex[2][3][8][32];
  __shared__ uint32_t part[2][8][32];  // warp 0's cubes, warp 1's sums
  __shared__ uint32_t hashes[8][32];
  const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  int cur = 0;
  auto put_to = [&](uint32_t (&s)[8][32], const Felt& x) {
#pragma unroll
    for (int q = 0; q < 8; q++) s[q][lane] = x.v[q];
  };
  auto get_from = [&](const uint32_t (&s)[8][32]) {
    Felt x;
#pragma unroll
    for (int q = 0; q < 8; q++) x.v[q] = s[q][lane];
    return x;
  };
  auto put = [&](const Felt& x) { put_to(ex[cur][w], x); };
  auto get = [&](uint32_t e) { return get_from(ex[cur][e]); };
  // Barriers of warps 0 and 1 (__syncthreads is barrier 0): 1, a cube is there
  // (warp 0 arrives and goes on, warp 1 waits); 2, a sum is there (the other
  // way round). They alternate: a warp arrives at one only after a wait at the
  // other, which its partner reaches past its own wait at the first.
  auto bar_arrive = [](int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); };
  auto bar_sync = [](int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); };
  for (uint32_t L = log_size;; L--) {
    const uint32_t n = 1u << L, i = 32 * blockIdx.x + lane;
    Felt e;  // this warp's state element; s2 with its round's constant added
    if (w == 2) {
      e = ladd(P252_TWO, P252_FULL_RC[2]);
    } else if (L == log_size) {
      e = load_hash(prev, 2 * (size_t)(i < n ? i : 0) + w);
    } else {
#pragma unroll
      for (int q = 0; q < 8; q++) e.v[q] = hashes[q][(2 * lane + w) & 31u];
    }
#pragma unroll 1
    for (int r = 0; r < 8; r++) {
      e = w == 2 ? e : ladd(e, P252_FULL_RC[3 * r + w]);
      e = fcube(w == 2 ? 3 : 1, e);
      put(e);
      __syncthreads();
      // the MDS, an element per warp (bounds: mds())
      const Felt s0 = get(0), s1 = get(1), s2 = get(2);
      if (w == 0) e = lreduce(ladd(ladd(ladd(s0, s2), ladd(s0, s1)), s0));
      else if (w == 1) e = lreduce(lsub(ladd(s0, s2), s1));
      else e = lsub(lsub(ladd(ladd(s0, s1), P252_S2_NEXT[r < 4 ? r : 83 + r]), s2), s2);
      cur ^= 1;
      if (r == 3) {  // the partial rounds
        put(e);
        __syncthreads();
        if (w == 0) {
          Felt x = get(2);
#pragma unroll 1
          for (int k = 0; k < 83; k++) {
            uint32_t T[16];
            sqr_wide8(x, T);
            const Felt q = redc(T);
            bar_sync(2);
            const Felt sum = get_from(part[1]);
            const Felt y = fmul_k(3, x, q);
            put_to(part[0], y);
            bar_arrive(1);
            Felt y2;
            y2.v[0] = y.v[0] << 1;
#pragma unroll
            for (int j = 1; j < 8; j++) y2.v[j] = __funnelshift_l(y.v[j - 1], y.v[j], 1);
            x = lsub(sum, y2);
          }
          put_to(ex[cur ^ 1][2], x);
        } else if (w == 1) {
          Felt s0 = get(0), s1 = e;
#pragma unroll 1
          for (int k = 0; k < 83; k++) {
            put_to(part[1], ladd(ladd(s0, s1), P252_S2_NEXT[4 + k]));
            bar_arrive(2);
            bar_sync(1);
            const Felt y = get_from(part[0]);
            const Felt u = ladd(s0, y), v = ladd(s0, s1);
            const Felt a0 = ladd(ladd(u, v), s0), a1 = lsub(u, s1);
            s0 = lreduce(a0);
            s1 = lreduce(a1);
          }
          put_to(ex[cur ^ 1][0], s0);
          put_to(ex[cur ^ 1][1], s1);
        }
        cur ^= 1;
        __syncthreads();
        e = get(w);
        cur ^= 1;
      }
    }
    if (w == 0) {
      if (i < n) store_hash(L == log_size ? out : up.p[L], i, e);
#pragma unroll
      for (int q = 0; q < 8; q++) hashes[q][lane] = e.v[q];
    }
    if (!to_root || L == 0) return;
    __syncthreads();
  }
}

// A batch of permutations: states of 3 big-endian hashes each (tests).
__global__ void poseidon252_permute_kernel(const uint8_t* __restrict__ in, uint32_t n, uint8_t* __restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    Felt s[3] = {load_hash(in, 3 * (size_t)i), load_hash(in, 3 * (size_t)i + 1), load_hash(in, 3 * (size_t)i + 2)};
    hades(s);
#pragma unroll
    for (int j = 0; j < 3; j++) store_hash(out, 3 * (size_t)i + j, s[j]);
  }
}

// Up to here a level is at most two blocks per SM and bound by latency. The
// line could lie anywhere from 4096 to 16384 nodes (the hashing of a 2^16
// Wide-Fibonacci proof differs by 0.04 of 11.5 ms); a thread per node at every
// size took 14.25.
constexpr size_t P252_TRIO_NODES = 8192;

int poseidon252_commit_nodes(cudaStream_t st, uint32_t top_log, uint32_t* const* layers) {
  for (int L = (int)top_log - 1; L >= 0; L--) {
    const uint8_t* prev = (const uint8_t*)layers[L + 1];
    if (L > 5) {
      GS_TRY(poseidon252_commit_on_layer(st, (uint32_t)L, prev, Cols(), 0, (uint8_t*)layers[L]));
      continue;
    }
    for (int k = 0; k <= L; k++) GS_REQUIRE(((uintptr_t)layers[k] & 15) == 0, "hash buffers must be 16-byte aligned");
    Levels252 up{};
    for (int k = 0; k < L; k++) up.p[k] = (uint8_t*)layers[k];
    launch_after(poseidon252_trio_kernel, 1, 96, 0, st, (uint32_t)L, prev, (uint8_t*)layers[L], up, 1u);
    note_launch();
    GS_CUDA_TRY(cudaGetLastError());
    break;
  }
  return OK;
}

int poseidon252_commit_on_layer(cudaStream_t st, uint32_t log_size, const uint8_t* d_prev,
                                Cols cols, uint32_t n_cols, uint8_t* d_out) {
  GS_REQUIRE(log_size <= 30, "layer log size out of range");
  GS_REQUIRE(d_out != nullptr, "null output");
  GS_REQUIRE(n_cols == 0 || cols.given(), "null column table");
  GS_REQUIRE(((uintptr_t)d_out & 15) == 0 && ((uintptr_t)d_prev & 15) == 0, "hash buffers must be 16-byte aligned");
  const size_t n = (size_t)1 << log_size;
  if (d_prev && n_cols == 0 && n <= P252_TRIO_NODES) {
    launch_after(poseidon252_trio_kernel, (unsigned)((n + 31) / 32), 96, 0, st, log_size, d_prev, d_out, Levels252{},
                 0u);
    note_launch();
    GS_CUDA_TRY(cudaGetLastError());
    return OK;
  }
  size_t blocks = (n + 127) / 128;
  const size_t cap = (size_t)num_sms() * 16;
  if (blocks > cap) blocks = cap;
  launch_after(poseidon252_layer_kernel, (unsigned)blocks, 128, 0, st, log_size, d_prev, cols, n_cols, d_out);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}

int poseidon252_permute(cudaStream_t st, const uint8_t* d_in, uint32_t n, uint8_t* d_out) {
  if (n == 0) return OK;
  GS_REQUIRE(((uintptr_t)d_in & 15) == 0 && ((uintptr_t)d_out & 15) == 0, "state buffers must be 16-byte aligned");
  const uint32_t blocks = (n + 127) / 128;
  poseidon252_permute_kernel<<<blocks, 128, 0, st>>>(d_in, n, d_out);
  note_launch();
  GS_CUDA_TRY(cudaGetLastError());
  return OK;
}

}  // namespace gs

namespace gs {

// ------------------------------------------------ proof of work, Poseidon252
// GrindOps<Poseidon252Channel>::grind (prover/backend/simd/grind.rs:152-190;
// the reference's CUDA backend hands it to that CPU code, cuda/backend.rs:
// 52-56): prefixed = poseidon_hash_many([POW_PREFIX, digest, pow_bits]); the
// answer is the smallest nonce (hi << 32) | low, low < 2^14, hi = 0, 1, ...,
// whose poseidon_hash(prefixed, nonce) has at least pow_bits trailing zero
// bits in its low 128 bits.
constexpr uint32_t P252_POW_PREFIX = 0x12345678u;
constexpr uint32_t P252_GRIND_LOW_LOG = 14, P252_GRIND_STEP = 128;

__device__ __forceinline__ Felt small_felt(uint32_t lo, uint32_t hi) {
  Felt x{};
  x.v[0] = lo;
  x.v[1] = hi;
  return to_mont(x);
}

// One thread: poseidon_hash_many of three values (two permutations).
__global__ void poseidon252_pow_prefix_kernel(const uint8_t* __restrict__ digest, uint32_t pow_bits,
                                              uint8_t* __restrict__ out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Felt s[3] = {};
  for (int b = 0; b < 2; b++) {
    if (b == 0) {
      s[0] = fadd(s[0], small_felt(P252_POW_PREFIX, 0));
      s[1] = fadd(s[1], load_hash(digest, 0));
    } else {
      s[0] = fadd(s[0], small_felt(pow_bits, 0));
      s[1] = fadd(s[1], P252_ONE);
    }
    hades(s);
  }
  store_hash(out, 0, s[0]);
}

// Persistent grid over 128-nonce steps of high words [hi0, hi0 + n_hi), in
// increasing nonce order; a block stops at the first step above the recorded
// minimum (a plain read, nothing waits), so the answer is still the smallest
// passing nonce (atomicMin over the 64-bit nonce).
__global__ void __launch_bounds__(P252_GRIND_STEP) poseidon252_grind_kernel(const uint8_t* __restrict__ prefixed,
                                                                           uint32_t hi0, uint32_t n_hi,
                                                                           uint32_t pow_bits,
                                                                           unsigned long long* result) {
  const volatile unsigned long long* best = result;
  const Felt pre = load_hash(prefixed, 0);
  constexpr uint32_t STEPS_PER_HI = (1u << P252_GRIND_LOW_LOG) / P252_GRIND_STEP;
  for (uint32_t step = blockIdx.x; step < n_hi * STEPS_PER_HI; step += gridDim.x) {
    const uint32_t hi = hi0 + step / STEPS_PER_HI;
    const uint32_t low0 = (step % STEPS_PER_HI) * P252_GRIND_STEP;
    if (*best < (((unsigned long long)hi << 32) | low0)) return;
    const uint32_t low = low0 + threadIdx.x;
    Felt s[3] = {pre, small_felt(low, hi), P252_TWO};
    hades(s);
    const Felt h = from_mont(s[0]);
    // trailing zeros of the low 128 bits (limbs 0..3)
    uint32_t tz = 128;
#pragma unroll
    for (int j = 3; j >= 0; j--)
      if (h.v[j]) tz = 32u * j + (uint32_t)(__ffs(h.v[j]) - 1);
    if (tz >= pow_bits) atomicMin(result, ((unsigned long long)hi << 32) | low);
  }
}

int poseidon252_grind(cudaStream_t st, const uint8_t* d_digest, uint32_t pow_bits, uint8_t* d_scratch,
                      uint32_t* h_word, uint64_t* nonce_out, bool digest_is_prefixed) {
  GS_REQUIRE(pow_bits <= 128, "pow_bits > 128 is not supported");
  GS_REQUIRE(((uintptr_t)d_digest & 15) == 0 && ((uintptr_t)d_scratch & 15) == 0, "buffers must be 16-byte aligned");
  const uint8_t* d_pre = d_digest;
  unsigned long long* d_res = reinterpret_cast<unsigned long long*>(d_scratch + 32);  // 8 bytes
  if (!digest_is_prefixed) {  // one thread, two permutations
    d_pre = d_scratch;        // 32 bytes
    poseidon252_pow_prefix_kernel<<<1, 32, 0, st>>>(d_digest, pow_bits, d_scratch);
    note_launch();
    GS_CUDA_TRY(cudaGetLastError());
  }
  // high words per launch: about twice the expected number of chunks
  // (2^(pow_bits - 14) each), 1 to 64
  const uint32_t e = pow_bits > P252_GRIND_LOW_LOG ? pow_bits - P252_GRIND_LOW_LOG + 1 : 0;
  const uint32_t n_hi = e >= 6 ? 64u : 1u << e;
  const uint32_t steps = n_hi * ((1u << P252_GRIND_LOW_LOG) / P252_GRIND_STEP);
  const uint32_t cap = 8u * (uint32_t)num_sms();
  const unsigned blocks = steps < cap ? steps : cap;
  // Bounded search: 2^20 high words cover pow_bits far beyond 40 with
  // overwhelming probability; running out is reported, never looped on.
  for (uint32_t hi = 0; hi < (1u << 20); hi += n_hi) {
    GS_CUDA_TRY(cudaMemsetAsync(d_res, 0xff, 8, st));
    poseidon252_grind_kernel<<<blocks, P252_GRIND_STEP, 0, st>>>(d_pre, hi, n_hi, pow_bits, d_res);
    note_launch();
    GS_CUDA_TRY(cudaGetLastError());
    GS_CUDA_TRY(cudaMemcpyAsync(h_word, d_res, 8, cudaMemcpyDeviceToHost, st));
    GS_TRY(stream_sync(st));
    uint64_t found;
    memcpy(&found, h_word, 8);
    if (found != ~0ull) {
      *nonce_out = found;
      return OK;
    }
  }
  set_error("poseidon252 grind: no nonce found within the search bound");
  return ERR_TIMEOUT;
}

}  // namespace gs
