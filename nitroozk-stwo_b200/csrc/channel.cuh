// Device-side Fiat-Shamir step of the Blake2s channel (Blake2sChannel::
// mix_root followed by draw_secure_felt, crates/stwo/src/core/channel/
// blake2s.rs), run at the end of a tree's launch (merkle_tree_kernel, the legacy
// merkle_tail_kernel) and between the layers of the fused FRI tail. Run by one
// warp, four lanes per compression.
//
//   mix_root:    digest <- Blake2s(digest || root), n_draws <- 0
//   draw_u32s:   Blake2s(digest || n_draws (LE u32) || 0x00), n_draws += 1
//   draw_felt:   repeat draw_u32s until all 8 words are < 2p; the secure
//                field element is the first 4 words reduced mod p.
//
// state: 8 digest words, n_draws, status (set nonzero when no challenge was
// found within the draw bound). felt_out: the challenge, then its square.
#pragma once
#include "runtime.cuh"
#include "blake2s.cuh"

namespace gs {

// One warp runs the step with four lanes per compression (blake2s_quad); its
// messages lie in shared memory.
struct ChannelWords {
  uint4 mix[4];   // digest, root
  uint4 draw[4];  // digest, draws so far, zeros
  uint4 felt;     // the challenge
};
constexpr uint32_t CHANNEL_MIX_BYTES = 64, CHANNEL_DRAW_BYTES = 37;

// Warp 0, before the root is known.
__device__ __forceinline__ void channel_begin(ChannelWords& w, const uint32_t* state) {
  const uint32_t lane = threadIdx.x;
  if (lane < 8) reinterpret_cast<uint32_t*>(w.mix)[lane] = state[lane];
  if (lane < 8) reinterpret_cast<uint32_t*>(w.draw)[8 + lane] = 0;
}
// Words j and 4 + j of the root, from lanes j < 4 of warp 0.
__device__ __forceinline__ void channel_root(ChannelWords& w, uint32_t j, uint32_t h0, uint32_t h1) {
  uint32_t* m = reinterpret_cast<uint32_t*>(w.mix);
  m[8 + j] = h0;
  m[12 + j] = h1;
}
// The hash of the mix message, the new digest (lanes j < 4).
__device__ __forceinline__ void channel_mixed(ChannelWords& w, uint32_t j, uint32_t h0, uint32_t h1, uint32_t* state) {
  uint32_t *m = reinterpret_cast<uint32_t*>(w.mix), *d = reinterpret_cast<uint32_t*>(w.draw);
  m[j] = d[j] = state[j] = h0;
  m[4 + j] = d[4 + j] = state[4 + j] = h1;
  if (j == 0) d[8] = 0;
}
// The hash of the draw message after `draws` earlier ones, in every quad of
// warp 0: true when the draw is done (the felt taken, in w.felt and felt_out
// with its square, or given up), false when it goes on with draws + 1. A draw
// is rejected with probability < 2^-27; 64 rejections in a row do not happen
// for a hash, and running out is reported, never looped on.
__device__ __forceinline__ bool channel_drawn(ChannelWords& w, uint32_t h0, uint32_t h1, uint32_t draws,
                                              uint32_t* state, uint32_t* felt_out) {
  const uint32_t lane = threadIdx.x;
  const bool ok = __all_sync(0xffffffffu, h0 < 2u * P && h1 < 2u * P);
  if (!ok && draws + 1 < 64) {
    if (lane == 0) w.draw[2].x = draws + 1;
    __syncwarp();
    return false;
  }
  if (lane < 4) reinterpret_cast<uint32_t*>(&w.felt)[lane] = h0 >= P ? h0 - P : h0;
  __syncwarp();
  if (lane == 0) {
    state[8] = draws + 1;
    if (ok) {
      const qm31 a = qm_make(w.felt.x, w.felt.y, w.felt.z, w.felt.w), a2 = qm_mul(a, a);
      felt_out[0] = a.x.a; felt_out[1] = a.x.b; felt_out[2] = a.y.a; felt_out[3] = a.y.b;
      felt_out[4] = a2.x.a; felt_out[5] = a2.x.b; felt_out[6] = a2.y.a; felt_out[7] = a2.y.b;
    } else {
      state[9] = 1;
    }
  }
  return true;
}

}  // namespace gs
