// Device-side Fiat-Shamir step of the Blake2s channel (Blake2sChannel::
// mix_root followed by draw_secure_felt, crates/stwo/src/core/channel/
// blake2s.rs), shared by the stand-alone channel kernel and the fused FRI
// tail kernel. Run by one thread.
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

// The step is two compressions whose messages lie in shared memory, so that a
// kernel runs them through the same compression its tree levels use (one copy
// of the unrolled rounds stays in the instruction cache; a lone warp that runs
// into another copy waits for its instructions).
struct ChannelWords {
  uint4 mix[4];   // digest, root
  uint4 draw[4];  // digest, draws so far, zeros
};
constexpr uint32_t CHANNEL_MIX_BYTES = 64, CHANNEL_DRAW_BYTES = 37;

__device__ __forceinline__ void channel_begin(ChannelWords& w, const uint32_t* state) {  // one thread
  w.mix[0] = make_uint4(state[0], state[1], state[2], state[3]);
  w.mix[1] = make_uint4(state[4], state[5], state[6], state[7]);
  w.draw[3] = make_uint4(0, 0, 0, 0);
}
__device__ __forceinline__ void channel_root(ChannelWords& w, const uint32_t h[8]) {  // one thread
  w.mix[2] = make_uint4(h[0], h[1], h[2], h[3]);
  w.mix[3] = make_uint4(h[4], h[5], h[6], h[7]);
}
// h: the hash of the mix message, the new digest (one thread).
__device__ __forceinline__ void channel_mixed(ChannelWords& w, const uint32_t h[8], uint32_t* state) {
  w.mix[0] = w.draw[0] = make_uint4(h[0], h[1], h[2], h[3]);
  w.mix[1] = w.draw[1] = make_uint4(h[4], h[5], h[6], h[7]);
  w.draw[2] = make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int j = 0; j < 8; j++) state[j] = h[j];
}
// h: the hash of the draw message after `draws` earlier ones. The same answer
// in every thread that holds h: true when the draw is done (the felt taken, or
// given up), false when it goes on with draws + 1; `one_thread` stores. A draw
// is rejected with probability < 2^-27; 64 rejections in a row do not happen
// for a hash, and running out is reported, never looped on.
__device__ __forceinline__ bool channel_drawn(ChannelWords& w, const uint32_t h[8], uint32_t draws, bool one_thread,
                                              uint32_t* state, uint32_t* felt_out, qm31& a) {
  bool ok = true;
#pragma unroll
  for (int j = 0; j < 8; j++) ok = ok && h[j] < 2u * P;
  if (!ok && draws + 1 < 64) {
    if (one_thread) w.draw[2].x = draws + 1;
    return false;
  }
  a = qm_make(h[0] >= P ? h[0] - P : h[0], h[1] >= P ? h[1] - P : h[1], h[2] >= P ? h[2] - P : h[2],
              h[3] >= P ? h[3] - P : h[3]);
  if (one_thread) {
    if (ok) {  // the challenge, then its square
      const qm31 a2 = qm_mul(a, a);
      felt_out[0] = a.x.a; felt_out[1] = a.x.b; felt_out[2] = a.y.a; felt_out[3] = a.y.b;
      felt_out[4] = a2.x.a; felt_out[5] = a2.x.b; felt_out[6] = a2.y.a; felt_out[7] = a2.y.b;
    } else {
      state[9] = 1;
    }
    state[8] = draws + 1;
  }
  return true;
}

}  // namespace gs
