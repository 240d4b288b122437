// Bit-serial learning rule shared by the plain and multi-network kernels.
#pragma once
#include <cstdint>

#include "axon_device.cuh"

namespace axon {

// The clip band [bandLo, bandHi] as bit masks (all ones or zeros per bit of the bounds).
struct Band {
  uint32_t lo[4], hi[4];
};
__device__ __forceinline__ Band band_of(uint32_t lo, uint32_t hi) {
  Band b;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    b.lo[i] = 0u - ((lo >> i) & 1u);
    b.hi[i] = 0u - ((hi >> i) & 1u);
  }
  return b;
}

// bs_clip (src/axon.mm:389-420) with the bounds as masks: both comparisons with the values
// before the clip, as borrow chains from the lowest plane, then the two sets, the upper bound
// last. 24 logic operations a word and no branch; with the bounds as numbers every plane cost
// a uniform test and a branch as well.
__device__ __forceinline__ void band_clip(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, const Band& b) {
  uint32_t lt = ~a0 & b.lo[0], gt = a0 & ~b.hi[0];
  lt = (~a1 & b.lo[1]) | (~(a1 ^ b.lo[1]) & lt);
  gt = (a1 & ~b.hi[1]) | (~(a1 ^ b.hi[1]) & gt);
  lt = (~a2 & b.lo[2]) | (~(a2 ^ b.lo[2]) & lt);
  gt = (a2 & ~b.hi[2]) | (~(a2 ^ b.hi[2]) & gt);
  lt = (~a3 & b.lo[3]) | (~(a3 ^ b.lo[3]) & lt);
  gt = (a3 & ~b.hi[3]) | (~(a3 ^ b.hi[3]) & gt);
  a0 = (a0 & ~lt) | (b.lo[0] & lt); a0 = (a0 & ~gt) | (b.hi[0] & gt);
  a1 = (a1 & ~lt) | (b.lo[1] & lt); a1 = (a1 & ~gt) | (b.hi[1] & gt);
  a2 = (a2 & ~lt) | (b.lo[2] & lt); a2 = (a2 & ~gt) | (b.hi[2] & gt);
  a3 = (a3 & ~lt) | (b.lo[3] & lt); a3 = (a3 & ~gt) | (b.hi[3] & gt);
}

// One 32-synapse word of k_learn's update, src/axon.mm:466-488: co-active pairs are
// potentiated (phase 1), depressed ltdRep times (phase 2) or take the legacy rule
// (phase 0); optional heterosynaptic LTD; then the clip band on every lane. `C` is any
// configuration with the fields ltdRep, hetero and bandHi; `band` is its clip band.
template <class C>
__device__ __forceinline__ void learn_word(uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3, uint32_t sp,
                                           bool want, uint32_t phase, uint32_t t, const C& c, const Band& band,
                                           uint32_t& nLTP, uint32_t& nLTD) {
  const uint32_t co = want ? sp : 0u;
  if (phase == 1u) {
    bs_inc(a0, a1, a2, a3, co);
    nLTP += __popc(co);
  } else if (phase == 2u) {
    for (uint32_t r = 0; r < c.ltdRep; ++r) bs_dec(a0, a1, a2, a3, co);
    nLTD += __popc(co) * c.ltdRep;
  } else {
    bs_inc(a0, a1, a2, a3, co);
    bs_dec(a0, a1, a2, a3, (want && (t % 2u == 1u)) ? ~sp : 0u);
  }
  if (c.hetero != 0u && phase == 1u) bs_dec(a0, a1, a2, a3, want ? ~sp : 0u);
  if (c.bandHi != 0u) band_clip(a0, a1, a2, a3, band);
}

}  // namespace axon
