// Bit-plane batched readout: B trajectories of one trained network, lane = trajectory.
//
// Same contract as the batched readout of batch.cu (present() with learn = 0 of
// src/axon.mm:815-888 for every trajectory, T steps in one cooperative launch). The 32
// neurons of a column are the 32 bits of a word throughout:
//
//   phase 1  a task is one column and 32 trajectories, one per lane. A lane walks its own
//            trajectory's active branches of the column. An active group nearly always has
//            one nonzero spike word S (one winning column of its eight), and the branch's 32
//            row counts popc(W3 row & S) come as six bit planes at once: W3 is kept
//            transposed (planes.cuh), so the count is the word's precomputed row-count
//            planes minus a carry-save sum of the masks of the neurons that S leaves out (or
//            the sum of the masks S holds, whichever is fewer). The planes are added into
//            the lane's drive planes with ripple-carry logic operations: no population
//            counts, no counters in shared memory, no atomics, no barrier between tasks.
//            Column drives go to global memory; a column whose drive reaches the
//            trajectory's floor (mostly 5/8 of its threshold two steps back, cand_floor) is a
//            candidate: a bit per column, and its drive planes, are kept for phase 2.
//   barrier
//   phase 2  a group of warps per trajectory: the column threshold from the candidates (from
//            all drives, with the gated columns' planes recomputed, when fewer than `target`
//            recurrent columns reached the floor), the exact k-of-32 of a gated column by one
//            thread (a radix select on the planes), and the records of the next step's
//            spikes.
//   barrier
//
// Column tiles (40 KiB) are staged in shared memory by bulk copies into a ring of slots; a
// CTA owns a fixed set of columns and walks it forwards and backwards in turn, so that the
// last slots of a step are the first of the next without a copy and the L2 serves the columns
// read last. The trajectories of a column's tasks are sorted by their number of active
// branches (a counting sort, by the warp that finishes an earlier column), since a task lasts
// as long as its slowest lane: 5.2 branches on average against 8 unsorted. With few
// trajectories only a part of each tile is needed and phase 1 reads it through L2 instead
// (DIRECT).
//
// Bound: the integer pipes. The drive is about 110 logic operations, address computations and
// shared loads per (column, trajectory, spike word), a third of them in divergent lanes, where
// the population-count form (batch.cu) takes 32 AND, POPC and packed adds, and 16 shared
// atomics. 640 threads leave 96 registers a thread (896 threads spilled and took 8 % longer).
// The L2 form has 896 threads: it waits for its reads, not for the pipes.
// Measured per step, config C at load 60 (batch.cu / this): 69 / 16 us for one trajectory,
// 86 / 24 for 16, 96 / 47 for 64, 98 / 56 for 100, 111 / 78 for 200, 133 / 101 for 300, 213 /
// 162 for 512.
#pragma once
#include <cstdint>

#include "axon_device.cuh"
#include "batch_common.cuh"
#include "planes.cuh"
#include "theta.cuh"

namespace axon {

namespace {

constexpr uint32_t kPadByte = 38u * 4u;  // byte offset of a block's zero word
constexpr uint32_t kRecList = 12;        // positions a record lists
// record header: byte offset of the word's block in its tile (bits 0..10), flags, the mask
// of the group's nonzero words above this one (bits 24..31)
constexpr uint32_t kRecOff = 0x7FFu, kRecOnes = 1u << 11, kRecBits = 1u << 12, kRecLong = 1u << 13;
constexpr uint32_t kRecSlow = kRecOnes | kRecBits | kRecLong;

// Record of a nonzero spike word S, word w of its group: x = header; y, z, w = byte offsets
// of up to 12 masks to sum, padded with the zero word (kRecLong: w is in use), or with
// kRecBits the positions as the set bits of y. The sum is of the neurons that the word
// leaves out, and is subtracted from the row counts, or with kRecOnes of those it holds.
__device__ __forceinline__ uint4 make_rec(uint32_t w, uint32_t more, uint32_t S) {
  const bool ones = __popc(S) <= 16;
  uint32_t bits = ones ? S : ~S;
  const uint32_t n = (uint32_t)__popc(bits);
  uint4 r;
  r.x = w * (kPlaneBlk * 4u) | (ones ? kRecOnes : 0u) | (more << 24);
  if (n > kRecList) {
    r.x |= kRecBits;
    r.y = bits;
    r.z = r.w = 0u;
    return r;
  }
  if (n > 8u) r.x |= kRecLong;
  uint32_t v[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    v[q] = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t at = bits ? (uint32_t)(__ffs(bits) - 1) * 4u : kPadByte;
      bits &= bits - 1u;
      v[q] |= at << (8 * i);
    }
  }
  r.y = v[0]; r.z = v[1]; r.w = v[2];
  return r;
}

__device__ __forceinline__ void fa(uint32_t a, uint32_t b, uint32_t c, uint32_t& s, uint32_t& k) {
  s = a ^ b ^ c;
  k = (a & b) | (a & c) | (b & c);
}

// out bit s of lane l = bit l of lane s's word
__device__ __forceinline__ uint32_t transpose32(uint32_t v, uint32_t lane) {
#pragma unroll
  for (int i = 4; i >= 0; --i) {
    const uint32_t j = 1u << i;
    const uint32_t lo = j == 16u ? 0x0000FFFFu : j == 8u ? 0x00FF00FFu : j == 4u ? 0x0F0F0F0Fu : j == 2u ? 0x33333333u : 0x55555555u;
    // the bits kept: those whose index agrees with the lane in bit j; the partner's others,
    // moved by j places (a rotation: what wraps around falls on kept bits), take the rest
    const uint32_t up = 0u - ((lane >> i) & 1u), keep = lo ^ up;
    const uint32_t x = __shfl_xor_sync(kFull, v, j);
    v = (v & keep) | (__funnelshift_l(x, x, (j ^ up) - up) & ~keep);
  }
  return v;
}

// Words of a tile, by byte offset: in global memory (read through the non-coherent path) or
// in shared memory (32-bit addresses, so that an offset costs one addition).
struct GlobalTile {
  const char* p;
  __device__ __forceinline__ GlobalTile at(uint32_t off) const { return {p + off}; }
  __device__ __forceinline__ uint32_t ld(uint32_t off) const { return __ldg(reinterpret_cast<const uint32_t*>(p + off)); }
  __device__ __forceinline__ uint4 ld4(uint32_t off) const { return __ldg(reinterpret_cast<const uint4*>(p + off)); }
  __device__ __forceinline__ uint2 ld2(uint32_t off) const { return __ldg(reinterpret_cast<const uint2*>(p + off)); }
  // the word at byte offset: byte i of v
  template <int I>
  __device__ __forceinline__ uint32_t pick(uint32_t v) const { return ld((v >> (8 * I)) & 0xFFu); }
  static __device__ __forceinline__ uint4 rec(const uint4* p) { return *p; }
};
struct SharedTile {
  uint32_t a;
  __device__ __forceinline__ SharedTile at(uint32_t off) const { return {a + off}; }
  __device__ __forceinline__ uint32_t lds(uint32_t x) const {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(x));
    return v;
  }
  __device__ __forceinline__ uint32_t ld(uint32_t off) const { return lds(a + off); }
  __device__ __forceinline__ uint4 ld4(uint32_t off) const {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a + off));
    return v;
  }
  __device__ __forceinline__ uint2 ld2(uint32_t off) const {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a + off));
    return v;
  }
  static __device__ __forceinline__ uint4 rec(const uint4* p) { return __ldcg(p); }
  // byte i of v added to the address by one dot product with a unit vector
  template <int I>
  __device__ __forceinline__ uint32_t pick(uint32_t v) const { return lds(__dp4a(v, 1u << (8 * I), a)); }
};

// Counts of one spike word per row, as six bit planes, in the cases the main loop leaves out:
// a sum of the masks the word holds, more than eight masks, or the masks as a bit set.
template <class Tile>
__device__ __forceinline__ void word_counts(Tile t, uint4 r, uint32_t (&d)[6]) {
  uint32_t z[5] = {0u, 0u, 0u, 0u, 0u};
  auto add = [&](uint32_t k) {  // one mask more
#pragma unroll
    for (int i = 0; i < 4; ++i) { const uint32_t x = z[i] & k; z[i] ^= k; k = x; }
    z[4] ^= k;  // at most 16 masks
  };
  if (r.x & kRecBits) {
    for (uint32_t bits = r.y; bits; bits &= bits - 1u) add(t.ld(4u * ((uint32_t)__ffs(bits) - 1u)));
  } else {
    const uint32_t v[3] = {r.y, r.z, r.w};
    const int nq = (r.x & kRecLong) ? 3 : 2;
    for (int q = 0; q < nq; ++q) {
      const uint32_t x = q == 0 ? v[0] : q == 1 ? v[1] : v[2];
      add(t.template pick<0>(x));
      add(t.template pick<1>(x));
      add(t.template pick<2>(x));
      add(t.template pick<3>(x));
    }
  }
  if (r.x & kRecOnes) {
#pragma unroll
    for (int i = 0; i < 5; ++i) d[i] = z[i];
    d[5] = 0u;
    return;
  }
  const uint4 p = t.ld4(128u);
  const uint2 p2 = t.ld2(144u);
  const uint32_t P[6] = {p.x, p.y, p.z, p.w, p2.x, p2.y};
  uint32_t b = 0u;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    d[i] = P[i] ^ z[i] ^ b;
    b = (~P[i] & (z[i] | b)) | (z[i] & b);
  }
  d[5] = P[5] ^ b;
}

// Drive planes of one (column, trajectory): m = the column's branches whose group spikes (of
// which this lane takes one in 1 << ls, starting at the first left in m), tile and conn the
// column's W3P block and connection row, rec the trajectory's records. DT1: dthr <= 1, a
// branch is above threshold when any of its counts is nonzero. A = sum of the counts (modes
// 0, 1), M = number of branches at or above dthr.
template <class Tile, bool LIN, bool DT1>
__device__ __forceinline__ void accumulate(Tile tile, Tile conn, uint32_t m, uint32_t ls, const uint4* rec,
                                           uint32_t ngrp, uint32_t dthr, uint32_t (&A)[kPlanes],
                                           uint32_t (&M)[6]) {
#pragma unroll
  for (int i = 0; i < (int)kPlanes; ++i) A[i] = 0u;
#pragma unroll
  for (int i = 0; i < 6; ++i) M[i] = 0u;
  const uint32_t n0 = dthr == 0u ? kFull : 0u;
  uint32_t N = n0, C[9];
  if (!DT1) {
#pragma unroll
    for (int i = 0; i < 9; ++i) C[i] = 0u;
  }
  if (m == 0u) return;
  auto drop = [&]() {  // the branch taken and those of the trajectory's other lanes
    m &= m - 1u;
    if (ls) {
      m &= m - 1u;
      if (ls > 1u) { m &= m - 1u; m &= m - 1u; }
    }
  };
  uint32_t s = (uint32_t)__ffs(m) - 1u;
  drop();
  uint4 r = Tile::rec(rec + conn.ld(4u * s));
  bool last = false;
  // the next word's record, of the same group or of the next branch's
  auto fetch = [&](uint32_t more) {
    uint32_t at;
    if (more) {
      at = ngrp + 8u * conn.ld(4u * s) + (uint32_t)__ffs(more) - 1u;
    } else {
      last = m == 0u;
      if (last) return;
      s = (uint32_t)__ffs(m) - 1u;
      drop();
      at = conn.ld(4u * s);
    }
    r = Tile::rec(rec + at);
  };
  // a word's counts into the sums
  auto absorb = [&](uint32_t d0, uint32_t d1, uint32_t d2, uint32_t d3, uint32_t d4, uint32_t d5, uint32_t more) {
    uint32_t kA = 0u, x;
    if (LIN) {
      kA = A[0] & d0;
      A[0] ^= d0;
      fa(A[1], d1, kA, A[1], kA);
      fa(A[2], d2, kA, A[2], kA);
      fa(A[3], d3, kA, A[3], kA);
      fa(A[4], d4, kA, A[4], kA);
      fa(A[5], d5, kA, A[5], kA);
      x = A[6] & kA; A[6] ^= kA; kA = x;
      x = A[7] & kA; A[7] ^= kA; kA = x;
      x = A[8] & kA; A[8] ^= kA; kA = x;
    }
    // once the branch's last word is in: one more branch above threshold for the neurons in N
    uint32_t kM = 0u;
    if (DT1) {
      N |= (d0 | d1 | d2) | (d3 | d4 | d5);
      kM = more ? 0u : N;
      N = more ? N : n0;
    } else {
      uint32_t k = C[0] & d0;
      C[0] ^= d0;
      fa(C[1], d1, k, C[1], k);
      fa(C[2], d2, k, C[2], k);
      fa(C[3], d3, k, C[3], k);
      fa(C[4], d4, k, C[4], k);
      fa(C[5], d5, k, C[5], k);
#pragma unroll
      for (int i = 6; i < 9; ++i) { x = C[i] & k; C[i] ^= k; k = x; }
      if (more == 0u) {
        uint32_t gt = 0u, eq = kFull;
#pragma unroll
        for (int i = 8; i >= 0; --i) {
          const uint32_t kb = ((dthr >> i) & 1u) ? kFull : 0u;
          gt |= eq & C[i] & ~kb;
          eq &= ~(C[i] ^ kb);
          C[i] = 0u;
        }
        kM = dthr < 512u ? gt | eq : 0u;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) { x = M[i] & kM; M[i] ^= kM; kM = x; }
    if (kA | kM) {  // rare: counts past 512, or 16 branches
      if (LIN) {
#pragma unroll
        for (int i = 9; i < (int)kPlanes; ++i) { x = A[i] & kA; A[i] ^= kA; kA = x; }
      }
#pragma unroll
      for (int i = 4; i < 6; ++i) { x = M[i] & kM; M[i] ^= kM; kM = x; }
    }
  };
  do {
    const uint32_t h = r.x, more = h >> 24;
    const Tile blk = tile.at(s * (kPlaneTile * 4u) + (h & kRecOff));
    if (!(h & kRecSlow)) {
      const uint32_t m0 = blk.template pick<0>(r.y), m1 = blk.template pick<1>(r.y), m2 = blk.template pick<2>(r.y),
                     m3 = blk.template pick<3>(r.y), m4 = blk.template pick<0>(r.z), m5 = blk.template pick<1>(r.z),
                     m6 = blk.template pick<2>(r.z), m7 = blk.template pick<3>(r.z);
      const uint4 p = blk.ld4(128u);
      const uint2 p2 = blk.ld2(144u);
      fetch(more);
      uint32_t s0, s1, k0, k1, k3, t0, q0, z0;
      fa(m0, m1, m2, s0, k0);
      fa(m3, m4, m5, s1, k1);
      const uint32_t s2 = m6 ^ m7, k2 = m6 & m7;
      fa(s0, s1, s2, z0, k3);
      fa(k0, k1, k2, t0, q0);
      const uint32_t z1 = t0 ^ k3, q1 = t0 & k3, z2 = q0 ^ q1, z3 = q0 & q1;
      const uint32_t b1 = ~p.x & z0, b2 = (~p.y & (z1 | b1)) | (z1 & b1), b3 = (~p.z & (z2 | b2)) | (z2 & b2),
                     b4 = (~p.w & (z3 | b3)) | (z3 & b3), b5 = b4 & ~p2.x;
      absorb(p.x ^ z0, p.y ^ z1 ^ b1, p.z ^ z2 ^ b2, p.w ^ z3 ^ b3, p2.x ^ b4, p2.y ^ b5, more);
    } else {
      uint32_t d[6];
      word_counts(blk, r, d);
      fetch(more);
      absorb(d[0], d[1], d[2], d[3], d[4], d[5], more);
    }
  } while (!last);
}

// Per-neuron drive planes from the sums: D (in A) = A + bst * M (modes 0, 1) or M (mode 2).
template <bool LIN>
__device__ __forceinline__ void combine_planes(uint32_t (&A)[kPlanes], const uint32_t (&M)[6], uint32_t bst) {
  if (LIN) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (!((bst >> q) & 1u)) continue;  // uniform over the launch
      uint32_t k = 0u;
#pragma unroll
      for (int i = 0; i < 6; ++i) fa(A[q + i], M[i], k, A[q + i], k);
#pragma unroll
      for (int i = q + 6; i < (int)kPlanes; ++i) { const uint32_t x = A[i] & k; A[i] ^= k; k = x; }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 6; ++i) A[i] = M[i];
  }
}

// D + the drive planes at p
__device__ __forceinline__ void add_planes(uint32_t (&D)[kPlanes], const uint4* p) {
  const uint4 a = __ldcg(p), b = __ldcg(p + 1), c = __ldcg(p + 2), e = __ldcg(p + 3);
  const uint32_t P[kPlanes] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w, e.x, e.y};
  uint32_t k = 0u;
#pragma unroll
  for (int i = 0; i < (int)kPlanes; ++i) fa(D[i], P[i], k, D[i], k);
}

// D minus the bias, saturating at zero
__device__ __forceinline__ void subtract_bias(uint32_t (&D)[kPlanes], const uint32_t* biasP) {
  uint32_t b = 0u;
#pragma unroll
  for (int i = 0; i < (int)kPlanes; ++i) {
    const uint32_t p = __ldg(biasP + i), x = D[i];
    D[i] = x ^ p ^ b;
    b = (~x & (p | b)) | (p & b);
  }
#pragma unroll
  for (int i = 0; i < (int)kPlanes; ++i) D[i] &= ~b;
}

// sum over the neurons in `mask` of the drives held in planes D
__device__ __forceinline__ uint32_t plane_sum(const uint32_t (&D)[kPlanes], uint32_t mask) {
  uint32_t s = 0u;
#pragma unroll
  for (int i = 0; i < 9; ++i) s += (uint32_t)__popc(D[i] & mask) << i;
  if (D[9] | D[10] | D[11] | D[12] | D[13]) {
#pragma unroll
    for (int i = 9; i < (int)kPlanes; ++i) s += (uint32_t)__popc(D[i] & mask) << i;
  }
  return s;
}

// value of rank `need` - 1 (descending) among the neurons in `cand`; on return cand = the
// neurons that hold it, win = those above it, need = how many of cand rank below the limit
__device__ __forceinline__ uint32_t plane_select(const uint32_t (&D)[kPlanes], uint32_t& cand, uint32_t& win,
                                                 uint32_t& need) {
  uint32_t v = 0u;
#pragma unroll
  for (int i = (int)kPlanes - 1; i >= 0; --i) {
    const uint32_t t = cand & D[i], n = (uint32_t)__popc(t);
    if (n >= need) {
      cand = t;
      v |= 1u << i;
    } else {
      win |= t;
      need -= n;
      cand &= ~t;
    }
  }
  return v;
}

// Exact k-of-32 on bit planes (src/axon.mm:134-144), by one thread: the radix select of the
// k-th largest drive leaves the larger ones and the neurons tied at it, of which the lowest
// lanes win. vk and, when asked for, vk1 are the values ranked k-1 and k (see warp_kwta).
__device__ __forceinline__ uint32_t plane_kwta(const uint32_t (&D)[kPlanes], uint32_t k, bool next, uint32_t& vk,
                                               uint32_t& vk1) {
  vk = vk1 = 0u;
  if (k == 0u) return 0u;
  if (k > 32u) return kFull;
  uint32_t cand = kFull, win = 0u, need = k;
  vk = plane_select(D, cand, win, need);
  if (next && k < 32u) {
    if ((uint32_t)__popc(cand) > need) {
      vk1 = vk;
    } else {
      uint32_t rest = ~(win | cand), w2 = 0u, one = 1u;
      vk1 = plane_select(D, rest, w2, one);
    }
  }
  for (; need; --need) {
    const uint32_t low = cand & (0u - cand);
    win |= low;
    cand ^= low;
  }
  return win;
}

// The smallest drive that makes a column of step t a candidate, from the trajectory's last
// two thresholds. Thresholds of trained networks move with period one while the inputs are
// clamped and mostly with period two (high, low) when they run free, so 5/8 of the threshold
// two steps back is nearly always reached by the `target` columns that are needed and by few
// more (100 to 250 columns in all on trained networks of 4,096; at 3/4 one trajectory in 200
// missed it each step, at 1/2 there are 180 to 490). At step 2 and two steps after the clamp
// (where it rises) the previous threshold serves instead, and at the first step after the
// clamp, where the drive of the inputs is missing, a sixth of it. At step 1 there is none: no column is a candidate and
// phase 2 selects from all drives.
__device__ __forceinline__ uint32_t cand_floor(const uint32_t* thPrev, uint32_t stride, uint32_t b, uint32_t t,
                                               uint32_t clampSteps, const PlanesCfg& c) {
  if (c.allCand) return 1u;
  if (t <= 1u) return t ? 0xFFFFFFFFu : 1u;
  const bool drop = t == clampSteps + 1u && !c.slabAlways;
  const bool next = t == clampSteps + 2u, one = drop || next || t == 2u;
  const uint32_t x = min(__ldcg(thPrev + ((t & 1u) ^ (one ? 1u : 0u)) * stride + b), 1u << 24);
  return max(drop ? x / 6u : next ? (7u * x) >> 3 : (5u * x) >> 3, 1u);
}

// Column threshold (k_topk, src/axon.mm:259-352) over the packed (drive << 13 | column)
// values val(0 .. n-1) of recurrent columns with a drive of at least lo >= 1: the need-th largest
// drive, 0 when fewer than `need` qualify. A radix select over the drives' distance from lo,
// at most 8 bits a pass. sH: 256 words, sR: 64. Every thread of the group calls it.
template <class V>
__device__ __forceinline__ uint32_t cand_theta(V val, uint32_t n, uint32_t incols, uint32_t lo,
                                               uint32_t need, uint32_t* sH, uint32_t* sR, WarpGrp g) {
  const uint32_t tid = g.tid(), lane = tid & 31u, warp = tid >> 5, nw = g.n() >> 5;
  uint32_t mx = 0u, cnt = 0u;
  for (uint32_t e = tid; e < n; e += g.n()) {
    const uint32_t p = val(e), s = p >> 13;
    if ((p & 8191u) >= incols && s >= lo) { mx = max(mx, s); ++cnt; }
  }
  mx = __reduce_max_sync(kFull, mx);
  cnt = __reduce_add_sync(kFull, cnt);
  if (lane == 0) { sR[warp] = mx; sR[32 + warp] = cnt; }
  for (uint32_t i = tid; i < 256u; i += g.n()) sH[i] = 0u;
  g.sync();
  const uint32_t Mx = __reduce_max_sync(kFull, lane < nw ? sR[lane] : 0u);
  const uint32_t count = __reduce_add_sync(kFull, lane < nw ? sR[32 + lane] : 0u);
  if (count < need) { g.sync(); return 0u; }
  const uint32_t nb = 32u - __clz(max(Mx - lo, 1u));
  uint32_t hi = nb, shift = nb > 8u ? nb - 8u : 0u, prefix = 0u, rem = need;
  for (;;) {
    const uint32_t dmask = (1u << (hi - shift)) - 1u;
    for (uint32_t e = tid; e < n; e += g.n()) {
      const uint32_t p = val(e), s = p >> 13;
      if ((p & 8191u) < incols || s < lo) continue;
      const uint32_t x = s - lo;
      if ((x >> hi) == (prefix >> hi)) atomicAdd(&sH[(x >> shift) & dmask], 1u);
    }
    g.sync();
    if (warp == 0u) {  // the bin where the count from the top reaches rem; then clear the bins
      uint32_t h[8], ls = 0u;
#pragma unroll
      for (int i = 0; i < 8; ++i) { h[i] = sH[lane * 8 + i]; ls += h[i]; }
      uint32_t S = ls;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t v = __shfl_down_sync(kFull, S, off);
        if (lane + off < 32u) S += v;
      }
      uint32_t cum = __shfl_down_sync(kFull, S, 1);
      if (lane == 31u) cum = 0u;
      if (S >= rem && cum < rem) {
        uint32_t b = lane * 8u;
#pragma unroll
        for (int i = 7; i >= 0; --i) {
          if (cum + h[i] >= rem) { b = lane * 8u + (uint32_t)i; break; }
          cum += h[i];
        }
        sR[62] = b;
        sR[63] = cum;
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) sH[lane * 8 + i] = 0u;
    }
    g.sync();
    prefix |= sR[62] << shift;
    rem -= sR[63];
    if (shift == 0u) break;
    hi = shift;
    shift = shift > 8u ? shift - 8u : 0u;
  }
  g.sync();
  return prefix + lo;
}

__device__ __forceinline__ void store_planes(uint4* p, const uint32_t (&D)[kPlanes]) {
  __stcg(p, make_uint4(D[0], D[1], D[2], D[3]));
  __stcg(p + 1, make_uint4(D[4], D[5], D[6], D[7]));
  __stcg(p + 2, make_uint4(D[8], D[9], D[10], D[11]));
  __stcg(p + 3, make_uint4(D[12], D[13], 0u, 0u));
}


// Drive planes of one (column, trajectory) outside phase 1, read through L2 and stored at p
// (after a threshold below the trajectory's floor, and there only). Out of line: its
// registers would add to phase 2's.
template <bool LIN, bool DT1>
__device__ __noinline__ void recompute_planes(const PlanesNet& net, const PlanesCfg& c, const uint32_t* act, uint32_t b,
                                              uint32_t col, const uint4* rec, const uint32_t* biasP, uint4* p) {
  const uint32_t ngrp = c.ncol / 8u;
  uint32_t m = 0u, D[kPlanes], M[6];
#pragma unroll 8
  for (uint32_t s = 0; s < 32u; ++s) {
    const uint32_t g = __ldg(net.conn + col * kNslot + s);
    m |= ((__ldcg(act + g * net.astr + (b >> 5)) >> (b & 31u)) & 1u) << s;
  }
  accumulate<GlobalTile, LIN, DT1>(GlobalTile{reinterpret_cast<const char*>(net.W3P + (size_t)col * kPlaneCol)},
                                   GlobalTile{reinterpret_cast<const char*>(net.conn + col * kNslot)}, m, 0u, rec, ngrp,
                                   c.dthr, D, M);
  combine_planes<LIN>(D, M, c.bst);
  if (biasP) subtract_bias(D, biasP);
  store_planes(p, D);
}

__host__ __device__ inline uint32_t group_words(uint32_t ncol) {
  return (ncol < kPlanesVals ? ncol : kPlanesVals) + ncol / 8u + 256u + 64u + 2u * kPlanesList;
}
// a list slot: per trajectory (whole blocks of 32) its active branches; the trajectories'
// order, as 16-bit values; 36 words of counts
__host__ __device__ inline uint32_t list_words(uint32_t nblk) { return 48u * nblk + 36u; }
constexpr uint32_t kMaxNS = 4, kMaxNL = 8;  // tile and list slots
// phase 1's tables: activity words, floors, state slots, lists
__host__ __device__ inline uint32_t table_words(uint32_t ncol, uint32_t nblk, uint32_t nl, bool serve) {
  return ncol / 8u * nblk + (serve ? 64u : 32u) * nblk + nl * list_words(nblk);
}
constexpr uint32_t kCtlWords = 2u * (kMaxNS + 2u * kMaxNL) + 4u + 2u * kMaxNS + 2u * kMaxNL;

}  // namespace

// SERVE: the recall server's form. The grid is cut into teams of CTAs, one per network, each
// with a barrier of its own; trajectory b of a team is at a step of its own, its state in a
// slot that stays its own from launch to launch (records, thresholds, candidate bits; the
// activity words are the network's), and it may end before the launch's last step.
template <bool LIN, bool DT1, bool DIRECT, bool SERVE>
__global__ void __launch_bounds__(planes_threads(DIRECT), 1) k_recall_planes(const __grid_constant__ PlanesDev d,
                                                                     const __grid_constant__ PlanesCfg c) {
  extern __shared__ __align__(128) uint32_t sm[];
  uint32_t team = 0;
  const uint64_t began = SERVE && threadIdx.x == 0 ? globaltimer_ns() : 0ull;
  if (SERVE)
    while (team + 1u < d.nteams && blockIdx.x >= d.teams[team + 1u].cta0) ++team;
  PlanesNet netS{};
  if (SERVE) netS = d.teams[team].net;
  const PlanesNet& net = SERVE ? netS : d.net;
  const uint32_t B = SERVE ? d.teams[team].B : c.B, G = SERVE ? d.teams[team].ncta : gridDim.x;
  const uint32_t cta = SERVE ? blockIdx.x - d.teams[team].cta0 : blockIdx.x;
  const uint32_t ncol = c.ncol, incols = c.incols, ngrp = ncol / 8u, nblk = (B + 31u) / 32u, Bp = 32u * nblk;
  const uint32_t nsl = c.nsl, nll = c.nll, NS = 1u << nsl, NL = 1u << nll;  // tile and list slots (none exist when DIRECT)
  uint32_t* sTile = sm;                       // [c.ns][kPlaneCol]
  uint32_t* sConn = sTile + c.ns * kPlaneCol;  // [c.ns][32] connection rows
  uint64_t* sBarT = reinterpret_cast<uint64_t*>(sConn + c.ns * 32u);  // [kMaxNS] a slot's tiles have landed
  uint64_t* sBarL = sBarT + kMaxNS;                                   // [kMaxNL] a slot's list is made
  uint64_t* sBarE = sBarL + kMaxNL;                                   // [kMaxNL] the column's tasks are done
  uint32_t* sMisc = reinterpret_cast<uint32_t*>(sBarE + kMaxNL);      // [0] barrier flag, [1..2] task counters, [3] give up
  uint32_t* sDone = sMisc + 4;          // [kMaxNL] finished tasks of the column in a list slot
  uint32_t* sCopies = sDone + kMaxNL;   // [kMaxNS] copies issued into a tile slot
  uint32_t* sFirst = sCopies + kMaxNS;  // [kMaxNS] number of the copy that the step's first column in the slot uses
  uint32_t* sMade = sFirst + kMaxNS;    // [kMaxNL] lists begun in a list slot
  // phase 1's tables and phase 2's groups share the rest
  uint32_t* sAct = sMade + kMaxNL;      // [ngrp][nblk] activity words of the step (every warp of every CTA reads
                                        // them: from global memory a few L2 lines would serve them all)
  uint32_t* sFloor = sAct + ngrp * nblk;  // [Bp] candidate floors
  uint32_t* sSlot = sFloor + Bp;          // [Bp] SERVE: state slots (kNoSlot: none, or at its end)
  uint32_t* sLists = sSlot + (SERVE ? Bp : 0u);  // [c.nl][list_words]
  uint32_t* sGrp = sAct;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nw = blockDim.x >> 5;
  const uint32_t ncols = cta < ncol ? (ncol - cta + G - 1u) / G : 0u;  // columns cta, cta + G, ...
  // lanes per trajectory in phase 1 (1 << ls), each on its own share of the active branches
  const bool sorted = !DIRECT || (nblk > 1u && ncols <= c.nl);
  const uint32_t ls = c.ls, tpw = 32u >> ls, ntb = sorted ? nblk << ls : (B + tpw - 1u) / tpw, ntask = ncols * ntb;
  const uint32_t part = lane & ((1u << ls) - 1u);
  const uint32_t ntbInv = (uint32_t)((0x100000000ull + ntb - 1u) / ntb);  // k / ntb of a task by a product (exact while k * ntb < 2^32: at most 8,192 columns x 16 tasks)

  if (tid == 0) {
    for (uint32_t i = 0; i < kMaxNS + kMaxNL; ++i) mbar_init(&sBarT[i], 1);
    for (uint32_t i = 0; i < kMaxNL; ++i) mbar_init(&sBarE[i], ntb);
    fence_proxy_async_smem();
  }
  for (uint32_t i = tid; i < 4u + 2u * kMaxNS + 2u * kMaxNL; i += blockDim.x) sMisc[i] = 0u;
  __syncthreads();

  const bool moved = SERVE && d.teams[team].moved != 0u;
  auto lane_before = [&](uint32_t b) -> uint32_t {
    const uint32_t ei = b < B ? __ldg(net.lanes + b) : kNoSlot;
    return ei != kNoSlot ? d.entries[ei].from : kNoSlot;
  };

  // a warp brings column ci of the CTA into a tile slot: the connection row by its lanes, the tiles by one bulk copy
  auto fill = [&](uint32_t slot, uint32_t ci) {
    const uint32_t col = cta + ci * G;
    sConn[slot * 32u + lane] = __ldg(net.conn + col * kNslot + lane);
    __syncwarp();
    if (lane == 0) {
      sCopies[slot] += 1u;
      fence_proxy_async_smem();
      mbar_expect_tx(&sBarT[slot], kPlaneCol * 4u);
      bulk_g2s(sTile + slot * kPlaneCol, net.W3P + (size_t)col * kPlaneCol, kPlaneCol * 4u, &sBarT[slot]);
    }
  };
  // and lists the trajectories for a column: each one's active branches (the activity words of
  // the column's 32 groups, transposed), the trajectories by falling number of them, so that
  // the 32 lanes of a task have nearly equal work
  auto conn_row = [&](uint32_t ci) { return __ldg(net.conn + (cta + ci * G) * kNslot + lane); };
  auto list = [&](uint32_t slot, uint32_t g, uint32_t skip) {
    uint32_t* sM = sLists + slot * list_words(nblk);
    uint16_t* sOrd = reinterpret_cast<uint16_t*>(sM + Bp);
    uint32_t* sCount = sM + 48u * nblk;  // [33]
    const uint32_t* row = sAct + g * nblk;
    sCount[lane] = 0u;
    if (lane == 0) sCount[32] = 0u;
    __syncwarp();
    // several blocks at a time, their loads, transposes and stores in groups: taken one by one
    // (the stores keep the next block's load behind them) a list of ten blocks took 4 us
    constexpr uint32_t kU = DIRECT ? 2 : 5;
    for (uint32_t k0 = 0; k0 < nblk; k0 += kU) {
      uint32_t m[kU];
#pragma unroll
      for (uint32_t i = 0; i < kU; ++i) m[i] = k0 + i < nblk && g >= skip ? row[k0 + i] : 0u;
#pragma unroll
      for (uint32_t i = 0; i < kU; ++i) m[i] = transpose32(m[i], lane);
#pragma unroll
      for (uint32_t i = 0; i < kU; ++i)
        if (k0 + i < nblk) {
          sM[32u * (k0 + i) + lane] = m[i];
          atomicAdd(sCount + __popc(m[i]), 1u);
        }
    }
    __syncwarp();
    const uint32_t n = sCount[32u - lane];
    uint32_t at = n;  // trajectories with at least 32 - lane active branches
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t x = __shfl_up_sync(kFull, at, off);
      if (lane >= (uint32_t)off) at += x;
    }
    __syncwarp();
    sCount[32u - lane] = at - n;
    if (lane == 31u) sCount[0] = at;
    __syncwarp();
    for (uint32_t k0 = 0; k0 < nblk; k0 += kU) {
      uint32_t o[kU];
#pragma unroll
      for (uint32_t i = 0; i < kU; ++i) o[i] = k0 + i < nblk ? (uint32_t)__popc(sM[32u * (k0 + i) + lane]) : 33u;
#pragma unroll
      for (uint32_t i = 0; i < kU; ++i)
        if (k0 + i < nblk) o[i] = atomicAdd(sCount + o[i], 1u);
#pragma unroll
      for (uint32_t i = 0; i < kU; ++i)
        if (k0 + i < nblk) sOrd[o[i]] = (uint16_t)(32u * (k0 + i) + lane);
    }
    __syncwarp();
    if (!DIRECT && lane == 0) {
      sMade[slot] += 1u;
      mbar_arrive(&sBarL[slot]);
    }
  };
  // copies this CTA issued must land before its shared memory is released
  auto drain = [&]() {
    __syncthreads();
    if (!DIRECT && tid < NS && sCopies[tid] != 0u)
      mbar_wait(&sBarT[tid], (sCopies[tid] - 1u) & 1u, c.waitNs > kDrainNs ? c.waitNs : kDrainNs);
    __syncthreads();
  };
  // tile slot of the step's q-th column: byte q % NS of slotMap, copy number sFirst[slot] +
  // q / NS of that slot; list slot q % NL, list number listBase(slot) + q / NL
  uint32_t slotMap = 0x03020100u, steps1 = 0;  // steps1: phase 1s run
  if (!DIRECT && warp < NS && warp < ncols) fill(warp, warp);

  bool back = false;  // direction of the walk over the CTA's columns
  uint32_t epoch = 0;
  for (uint32_t t = 0; t < c.T; ++t) {
    const uint32_t ap = (t + net.par) & 1u;
    const uint32_t* actIn = net.act + (size_t)ap * ngrp * net.astr;
    uint32_t* actOut = net.act + (size_t)(ap ^ 1u) * ngrp * net.astr;
    // Afferent cache. While the inputs are clamped their spikes are the cue at every step, so
    // the input groups' share of the drives is the same in steps 1..clampSteps. Step 1, whose
    // drives are that share alone (no recurrent column spikes at step 0), stores its planes;
    // the others leave the input groups out, half of the clamped steps' spike words, and add
    // the stored planes.
    const bool affStore = !SERVE && d.aff != nullptr && t == 1u;
    const bool affAdd = !SERVE && d.aff != nullptr && t >= 2u && t <= c.clampSteps;
    const uint32_t skip = affAdd ? incols / 8u : 0u;  // the groups below are left out
    // ---------------- phase 1 (nothing spikes before step 0: every drive is zero there)
    if (SERVE || t > 0u || d.refBall != nullptr) {
      uint32_t g0 = 0;  // the connection row of the warp's first list, on its way during the copies below
      if (!DIRECT && warp < NL && warp < ncols) g0 = conn_row(back ? ncols - 1u - warp : warp);
      if (SERVE && moved && t == 0u) {
        // the trajectories have other lanes than in the launch before: a warp takes a group's
        // old words, one per lane, and puts the new ones together bit by bit (about 3 us for
        // 512 groups)
        for (uint32_t b = tid; b < Bp; b += blockDim.x) sFloor[b] = lane_before(b);
        __syncthreads();
#pragma unroll 4
        for (uint32_t g = warp; g < ngrp; g += nw) {
          const uint32_t old = lane < net.astr ? __ldcg(actIn + g * net.astr + lane) : 0u;
          uint32_t mine = 0u;
          for (uint32_t k = 0; k < nblk; ++k) {
            const uint32_t f = sFloor[32u * k + lane], w = __shfl_sync(kFull, old, (f >> 5) & 31u);
            const uint32_t now = __ballot_sync(kFull, f != kNoSlot && ((w >> (f & 31u)) & 1u) != 0u);
            if (lane == k) mine = now;
          }
          if (lane < nblk) sAct[g * nblk + lane] = mine;
        }
        __syncthreads();
      } else if (SERVE) {
        for (uint32_t g = tid; g < ngrp; g += blockDim.x)
          for (uint32_t k = 0; k < nblk; ++k) sAct[g * nblk + k] = __ldcg(actIn + g * net.astr + k);
      }
      if (SERVE) {
        for (uint32_t b = tid; b < Bp; b += blockDim.x) {
          const uint32_t ei = b < B ? __ldg(net.lanes + b) : kNoSlot;
          uint32_t slot = kNoSlot, fl = 0xFFFFFFFFu;
          if (ei != kNoSlot) {
            const PlanesEntry e = d.entries[ei];
            if (e.t0 + t < e.steps) {
              slot = e.slot;
              fl = cand_floor(d.thPrev, d.thStride, slot, e.t0 + t, e.clamp, c);
            }
          }
          sSlot[b] = slot;
          sFloor[b] = fl;
        }
      } else {
        for (uint32_t i = tid; i < ngrp * nblk / 4u; i += blockDim.x)
          reinterpret_cast<uint4*>(sAct)[i] = __ldcg(reinterpret_cast<const uint4*>(actIn) + i);
        for (uint32_t b = tid; b < Bp; b += blockDim.x)
          sFloor[b] = b < B ? cand_floor(d.thPrev, d.thStride, b, t, c.clampSteps, c) : 0xFFFFFFFFu;
      }
      __syncthreads();
      if (!DIRECT && warp < NL && warp < ncols) list(warp, g0, skip);
      if (DIRECT && sorted) {  // every column's list at once
        for (uint32_t ci = warp; ci < ncols; ci += nw) list(ci, conn_row(ci), skip);
        __syncthreads();
      }
      // the next step's activity words, last read in step t-1
      for (uint32_t i = cta * blockDim.x + tid; i < ngrp * net.astr; i += G * blockDim.x) __stcg(actOut + i, 0u);
      for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(&sMisc[1u + (t & 1u)], 1u);
        k = __shfl_sync(kFull, k, 0);
        if (k >= ntask) break;
        const uint32_t q = ntb == 1u ? k : __umulhi(k, ntbInv), at = tpw * (k - q * ntb) + (lane >> ls);
        const uint32_t ci = back ? ncols - 1u - q : q, col = cta + ci * G;
        uint32_t slot = 0u, lslot = 0u, ln = 0u, b, m, A[kPlanes], M[6];
        if (DIRECT && sorted) {
          const uint32_t* sM = sLists + q * list_words(nblk);
          b = reinterpret_cast<const uint16_t*>(sM + Bp)[at];
          m = sM[b];
        } else if (DIRECT) {
          b = at;
          const uint32_t g = __ldg(net.conn + col * kNslot + lane);
          m = transpose32(g >= skip ? sAct[g * nblk + (b >> 5)] : 0u, lane);
          if (ls) m = __shfl_sync(kFull, m, b & 31u);
        } else {
          const uint32_t u = q >> nsl, lu = q >> nll;
          slot = (slotMap >> (8u * (q & (NS - 1u)))) & 0xFFu;
          lslot = q & (NL - 1u);
          // a task may be claimed several uses of its slots ahead: that copy and that list must
          // have begun before the parity of its phase means anything
          const uint32_t cp = sFirst[slot] + u;
          ln = steps1 * ((ncols - lslot + NL - 1u) >> nll) + lu;
          auto ready = [&]() {
            return ld_volatile(&sMade[lslot]) > ln && mbar_test(&sBarL[lslot], ln & 1u) &&
                   ld_volatile(&sCopies[slot]) > cp && mbar_test(&sBarT[slot], cp & 1u);
          };
          bool ok = ready();
          if (!ok) {
            const uint64_t t0 = globaltimer_ns();
            for (uint32_t it = 1; !ok; ++it) {
              __nanosleep(100);  // the polls would take issue slots from the warps that make the lists
              ok = ready();
              if ((it & 63u) == 0u && !ok && (ld_volatile(&sMisc[3]) != 0u || globaltimer_ns() - t0 > c.waitNs)) break;
            }
          }
          if (!__all_sync(kFull, ok)) {  // the copy did not land in time: the launch ends
            if (lane == 0) { atomicCAS(d.err, 0u, kErrTimeout); sMisc[3] = 1u; }
            break;
          }
          const uint32_t* sM = sLists + lslot * list_words(nblk);
          b = reinterpret_cast<const uint16_t*>(sM + Bp)[at];
          m = sM[b];
        }
        for (uint32_t i = 0; i < part; ++i) m &= m - 1u;
        const uint32_t sl = SERVE ? sSlot[b] : b;  // a lane without a trajectory has no active branch
        const uint4* recb = d.rec + (size_t)sl * (ngrp + ncol);
        if (DIRECT)
          accumulate<GlobalTile, LIN, DT1>(GlobalTile{reinterpret_cast<const char*>(net.W3P + (size_t)col * kPlaneCol)},
                                           GlobalTile{reinterpret_cast<const char*>(net.conn + col * kNslot)}, m, ls, recb,
                                           ngrp, c.dthr, A, M);
        else
          accumulate<SharedTile, LIN, DT1>(SharedTile{smem_u32(sTile + slot * kPlaneCol)},
                                           SharedTile{smem_u32(sConn + slot * 32u)}, m, ls, recb, ngrp, c.dthr, A,
                                           M);
        __syncwarp();
        uint32_t last = 0, gl = 0;
        if (!DIRECT) {  // the warp that finishes a column's last task refills its slots
          if (lane == 0) {
            mbar_arrive(&sBarE[lslot]);
            last = atomicAdd(&sDone[lslot], 1u) + 1u == ntb;
            if (last) mbar_wait(&sBarE[lslot], ln & 1u, c.waitNs);  // every arrival is made: orders the others' reads
          }
          last = __shfl_sync(kFull, last, 0);
          if (last && q + NL < ncols) gl = conn_row(back ? ncols - 1u - (q + NL) : q + NL);
          if (last && q + NS < ncols) fill(slot, back ? ncols - 1u - (q + NS) : q + NS);
        }
        for (uint32_t o = 1; o < (1u << ls); o <<= 1) {  // the sums of a trajectory's lanes
          uint32_t k2 = 0u;
          if (LIN) {
#pragma unroll
            for (int i = 0; i < (int)kPlanes; ++i) fa(A[i], __shfl_xor_sync(kFull, A[i], o), k2, A[i], k2);
          }
          k2 = 0u;
#pragma unroll
          for (int i = 0; i < 6; ++i) fa(M[i], __shfl_xor_sync(kFull, M[i], o), k2, M[i], k2);
        }
        combine_planes<LIN>(A, M, c.bst);
        if (!SERVE && part == 0u && b < B) {
          if (affStore) store_planes(d.aff + ((size_t)col * Bp + b) * 4u, A);
          if (affAdd) add_planes(A, d.aff + ((size_t)col * Bp + b) * 4u);
        }
        if (!SERVE && d.biasP) subtract_bias(A, d.biasP + col * 16u);
        const uint32_t s = plane_sum(A, kFull);
        if (part == 0u && (SERVE ? sl != kNoSlot : b < B)) {
          __stcg(d.drv + (size_t)sl * d.drvB + (size_t)col * d.drvC, s);
          if (!SERVE && d.refBall != nullptr && col >= incols) {  // driveLog of k_emit, src/axon.mm:216-220
            const uint32_t rb = __ldg(d.refBall + (size_t)b * ncol + col);
            const uint32_t sh = rb & __ldg(d.multM + col), ex = rb & ~sh;
            uint32_t* dl = d.driveLog + (size_t)b * 256u + t * 4u;
            if (sh) { atomicAdd(dl + 0, plane_sum(A, sh)); atomicAdd(dl + 1, (uint32_t)__popc(sh)); }
            if (ex) { atomicAdd(dl + 2, plane_sum(A, ex)); atomicAdd(dl + 3, (uint32_t)__popc(ex)); }
          }
          const bool cand = s >= sFloor[b];
          if (cand) atomicOr(d.candB + (size_t)sl * (ncol / 32u) + (col >> 5), 1u << (col & 31u));
          if (cand || (!SERVE && c.storeAll != 0u && s != 0u)) store_planes(d.candP + ((size_t)sl * ncol + col) * 4u, A);
        }
        if (last) {
          __syncwarp();
          if (lane == 0) sDone[lslot] = 0u;
          if (q + NL < ncols) list(lslot, gl, skip);
        }
      }
      __syncthreads();
      if (!DIRECT && sMisc[3] != 0u) { drain(); return; }
      if (tid == 0) sMisc[1u + (t & 1u)] = 0u;
      if (!DIRECT) {  // the slots' columns at the end of this step are the first of the next
        uint32_t map = 0u;
        if (tid < NS && tid < ncols) sFirst[(slotMap >> (8u * tid)) & 0xFFu] += ((ncols - tid + NS - 1u) >> nsl) - 1u;
        for (uint32_t r = 0; r < NS && r < ncols; ++r) map |= ((slotMap >> (8u * ((ncols - 1u - r) & (NS - 1u)))) & 0xFFu) << (8u * r);
        slotMap = map;
        back = !back;
        ++steps1;
      }
      if (!grid_barrier(net.bar, d.err, G, epoch++, c.waitNs, sMisc)) { drain(); return; }
    }

    // ---------------- phase 2
    const uint32_t NG = c.ng, gq = nw / NG, gx = nw % NG;
    const uint32_t gi = warp < gx * (gq + 1u) ? warp / (gq + 1u) : gx + (warp - gx * (gq + 1u)) / gq;
    const uint32_t gnw = gq + (gi < gx ? 1u : 0u), w0 = gi * gq + min(gi, gx);
    const WarpGrp grp{tid - 32u * w0, 32u * gnw, 1u + gi};
    const uint32_t nV = min(ncol, kPlanesVals);
    uint32_t* const sV = sGrp + gi * group_words(ncol);  // the first nV candidates: drive << 13 | column
    uint32_t* const sNz = sV + nV;                       // nonzero words of each presynaptic group
    uint32_t* const sH = sNz + ngrp;
    uint32_t* const sR = sH + 256u;                      // [0..63]; [61] gated columns
    uint32_t* const sList = sR + 64u;                    // gated entries
    uint32_t* const sBall = sList + kPlanesList;         // and their ballots
    for (uint32_t b = gi * G + cta; b < B; b += NG * G) {
      uint32_t sl = b, tl = t, tEnd = c.T, clampEnd = c.clampSteps, ncue = incols;  // state slot, own step, its bounds
      const uint32_t* cues = nullptr;
      uint32_t* fin = nullptr;  // where the final spikes go, in the last step
      if (SERVE) {
        const uint32_t ei = __ldg(net.lanes + b);
        if (ei == kNoSlot) continue;
        const PlanesEntry e = d.entries[ei];
        sl = e.slot;
        tl = e.t0 + t;
        tEnd = e.steps;
        clampEnd = e.clamp;
        ncue = e.ncue;
        cues = d.cues + e.cueOff;
        if (tl >= tEnd) continue;
        if (tl + 1u == tEnd) {
          fin = d.finalOut + (size_t)e.done * ncol;
          for (uint32_t i = grp.t; i < ncol / 4u; i += grp.nt) __stcg(reinterpret_cast<uint4*>(fin) + i, make_uint4(0u, 0u, 0u, 0u));
        }
      } else if (d.finalOut && t + 1u == c.T) {
        fin = d.finalOut + (size_t)b * ncol;
      }
      const bool clamp = tl < clampEnd;
      const uint32_t fl = cand_floor(d.thPrev, d.thStride, sl, tl, clampEnd, c), ncw = ncol / 32u;
      for (uint32_t i = grp.t; i < ngrp; i += grp.nt) sNz[i] = 0u;
      if (grp.t == 0) sR[60] = sR[61] = 0u;
      grp.sync();
      for (uint32_t i = grp.t; i < ncw; i += grp.nt) {  // the candidates' columns
        uint32_t x = __ldcg(d.candB + (size_t)sl * ncw + i);
        if (x == 0u) continue;
        __stcg(d.candB + (size_t)sl * ncw + i, 0u);
        for (uint32_t at = atomicAdd(&sR[60], (uint32_t)__popc(x)); x; x &= x - 1u, ++at)
          if (at < nV) sV[at] = 32u * i + (uint32_t)__ffs(x) - 1u;
      }
      grp.sync();
      uint32_t n = sR[60], theta = 1u;
      // too many candidates for the group's memory, or a threshold below the floor: the select
      // runs on all drives, and in the second case the gated columns' planes are recomputed
      bool redo = n > nV;
      uint4* candb = d.candP + (size_t)sl * ncol * 4u;
      uint32_t* candW = reinterpret_cast<uint32_t*>(candb);  // 16 words per column
      auto drive = [&](uint32_t cc) { return (__ldcg(d.drv + (size_t)sl * d.drvB + (size_t)cc * d.drvC) << 13) | cc; };
      auto val = [&](uint32_t e) -> uint32_t { return e < nV ? sV[e] : drive(e); };
      if (c.targetCols == 0u && c.topkPar == 0u) theta = 0xFFFFFFu;
      if (!redo) {
        for (uint32_t e = grp.t; e < n; e += grp.nt) sV[e] = drive(sV[e]);
        grp.sync();
        if (c.targetCols != 0u) {
          theta = cand_theta(val, n, incols, fl, c.targetCols, sH, sR, grp);
          redo = theta == 0u && fl > 1u;
        } else {
          redo = c.topkPar != 0u && fl > 1u;
        }
      }
      if (redo) {
        n = ncol;
        for (uint32_t cc = grp.t; cc < nV; cc += grp.nt) sV[cc] = drive(cc);
        grp.sync();
        if (c.targetCols != 0u) theta = cand_theta(val, n, incols, 1u, c.targetCols, sH, sR, grp);
      }
      const uint32_t gate = max(theta, 1u);
      const uint32_t* stimb = SERVE ? nullptr : d.stims + (size_t)b * ncol;
      uint4* recb = d.rec + (size_t)sl * (ngrp + ncol);
      // gated columns (clamped input columns take the cue instead)
      const uint32_t cMin = clamp ? incols : 0u;
      auto gated = [&](uint32_t p) { return (p >> 13) >= gate && (p & 8191u) >= cMin; };
      for (uint32_t e = grp.t; e < n; e += grp.nt)
        if (gated(val(e))) {
          const uint32_t i = atomicAdd(&sR[61], 1u);
          if (i < kPlanesList) sList[i] = e;
        }
      // the i-th word of the cue: its column, and its spikes
      auto cue_word = [&](uint32_t i, uint32_t& cc) -> uint32_t {
        cc = SERVE ? __ldg(cues + i) : i;
        return SERVE ? kFull : __ldg(stimb + i);
      };
      if (clamp)
        for (uint32_t i = grp.t; i < ncue; i += grp.nt) {
          uint32_t cc;
          if (cue_word(i, cc) != 0u) atomicOr(&sNz[cc >> 3], 1u << (cc & 7u));
        }
      grp.sync();
      const uint32_t npend = sR[61];
      // spikes of gated entry e: k-of-32, the k_emit counters (src/axon.mm:225-234), its group's mask
      auto spike = [&](uint32_t e) -> uint32_t {
        const uint32_t cc = val(e) & 8191u;
        uint32_t D[kPlanes], vk, vk1;
        const uint4* pp = candb + (size_t)cc * 4u;
        const uint4 a = __ldcg(pp), q = __ldcg(pp + 1), x = __ldcg(pp + 2), y = __ldcg(pp + 3);
        D[0] = a.x; D[1] = a.y; D[2] = a.z; D[3] = a.w; D[4] = q.x; D[5] = q.y; D[6] = q.z; D[7] = q.w;
        D[8] = x.x; D[9] = x.y; D[10] = x.z; D[11] = x.w; D[12] = y.x; D[13] = y.y;
        const uint32_t ball = plane_kwta(D, c.k, !SERVE && d.stats != nullptr, vk, vk1);
        if (!SERVE && d.stats != nullptr && ball != 0u && cc >= incols) {
          uint32_t* st = d.stats + (size_t)b * 1024u;
          const uint32_t sb = 64u + t * 8u;
          atomicAdd(st + 0, 1u);
          atomicAdd(st + 1, (uint32_t)__popc(ball));
          atomicAdd(st + sb + 0u, vk - vk1);
          atomicAdd(st + sb + 1u, vk);
          atomicAdd(st + sb + 2u, 1u);
          if (vk == vk1) atomicAdd(st + sb + 3u, 1u);
          if (vk == 0u) atomicAdd(st + sb + 4u, 1u);
        }
        if (ball != 0u) atomicOr(&sNz[cc >> 3], 1u << (cc & 7u));
        return ball;
      };
      // a nonzero spike word of column cc, once every group mask is complete
      auto emit = [&](uint32_t cc, uint32_t S) {
        if (!SERVE && d.hist) d.hist[((size_t)b * c.T + t) * ncol + cc] = S;
        if (fin) fin[cc] = S;
        if (tl + 1u >= tEnd) return;
        const uint32_t g = cc >> 3, w = cc & 7u, nz = sNz[g];
        const uint4 r = make_rec(w, (nz >> w >> 1) << w << 1, S);
        if ((nz & ((1u << w) - 1u)) == 0u) {
          __stcg(recb + g, r);
          atomicOr(actOut + g * net.astr + (b >> 5), 1u << (b & 31u));
        } else {
          __stcg(recb + ngrp + cc, r);
        }
      };
      // more gated columns than the list holds: all entries are walked and their spikes wait in global memory
      const bool over = npend > kPlanesList;
      const uint32_t walk = over ? n : npend;
      if (redo && gate < fl && c.storeAll == 0u)  // (at or above the floor they were stored)
        for (uint32_t i = grp.t; i < walk; i += grp.nt) {
          const uint32_t e = over ? i : sList[i];  // = the column
          if (over && !gated(val(e))) continue;
          const uint32_t bit = SERVE && moved && t == 0u ? lane_before(b) : b;  // its place in the activity words
          recompute_planes<LIN, DT1>(net, c, actIn, bit, e, recb, d.biasP ? d.biasP + e * 16u : nullptr, candb + (size_t)e * 4u);
        }
      for (uint32_t i = grp.t; i < walk; i += grp.nt) {
        const uint32_t e = over ? i : sList[i];
        if (over && !gated(val(e))) continue;
        const uint32_t S = spike(e);
        if (over) __stcg(candW + 16u * (val(e) & 8191u) + 15u, S);
        else sBall[i] = S;
      }
      grp.sync();
      // then the records, the clamped cue's after the gated columns'
      const uint32_t cue = clamp ? ncue : 0u;
      for (uint32_t i = grp.t; i < walk + cue; i += grp.nt) {
        uint32_t cc, S;
        if (i >= walk) {
          S = cue_word(i - walk, cc);
        } else {
          const uint32_t e = over ? i : sList[i], p = val(e);
          if (over && !gated(p)) continue;
          cc = p & 8191u;
          S = over ? __ldcg(candW + 16u * cc + 15u) : sBall[i];
        }
        if (S) emit(cc, S);
      }
      if (grp.t == 0) __stcg(d.thPrev + (tl & 1u) * d.thStride + sl, gate);
      grp.sync();
    }
    if (t + 1u == c.T) break;
    if (!grid_barrier(net.bar, d.err, G, epoch++, c.waitNs, sMisc)) { drain(); return; }
  }
  drain();
  if (SERVE && cta == 0u && tid == 0) d.teamNs[team] = (uint32_t)(globaltimer_ns() - began);
}


namespace {
size_t planes_smem(uint32_t ncol, uint32_t B, uint32_t ns, uint32_t nl, uint32_t ng, bool serve) {
  const size_t table = table_words(ncol, (B + 31u) / 32u, nl, serve), groups = (size_t)ng * group_words(ncol);
  return ((size_t)ns * (kPlaneCol + 32u) + kCtlWords + (table > groups ? table : groups)) * 4u;
}
template <bool LIN, bool DT1, bool SERVE>
const void* planes_fn2(uint32_t direct) {
  return direct ? (const void*)k_recall_planes<LIN, DT1, true, SERVE> : (const void*)k_recall_planes<LIN, DT1, false, SERVE>;
}
template <bool SERVE>
const void* planes_fn(const PlanesCfg& c, uint32_t direct) {
  if (c.mode == 2u) return c.dthr <= 1u ? planes_fn2<false, true, SERVE>(direct) : planes_fn2<false, false, SERVE>(direct);
  return c.dthr <= 1u ? planes_fn2<true, true, SERVE>(direct) : planes_fn2<true, false, SERVE>(direct);
}

// Shared-memory shares for at most B trajectories in one team, `cols` columns in one CTA and
// `want` phase-2 groups.
size_t planes_fit(uint32_t ncol, uint32_t B, bool direct, bool serve, uint32_t cols, uint32_t want, PlanesCfg* c) {
  constexpr size_t kLimit = 227u * 1024u;
  // lanes per trajectory: one, but a handful of trajectories would leave most lanes idle while
  // the others walk eight branches in a row (us per step at 1 / 8 / 16 / 24 trajectories of a
  // 4,096-column network: 21.3 / 24.5 / 27.3 / 30.5 with one lane, 18.1 / 21.0 / 24.6 / 31.5
  // with two, 16.6 / 19.6 / 26.6 / 32.7 with four)
  c->ls = B > 20u ? 0u : B > 10u ? 1u : 2u;
  // more, too, where one would leave most of a CTA's warps without a task (two columns of a
  // 256-column network and 40 trajectories are four tasks)
  while (direct && c->ls < 2u && cols * ((B + 31u) / 32u << (c->ls + 1u)) <= 28u) ++c->ls;
  c->ns = c->nl = 0;
  c->nsl = 2;
  c->nll = 3;
  c->ng = want < 3u ? want : 3u;
  auto bytes = [&]() { return planes_smem(ncol, B, c->ns, c->nl, c->ng, serve); };
  auto fits = [&]() { return bytes() <= kLimit; };
  if (!direct) {
    // within 195 KiB, where that is possible with four list slots, the L1 has 60 KiB instead of
    // 28, which the record gathers feel (us per step, 28 / 60 KiB: 107 / 101 at 300
    // trajectories, 111 / 102 at 320)
    constexpr size_t kRoomy = 195u * 1024u;
    c->ns = 1u << c->nsl;
    c->nl = 1u << c->nll;
    if (bytes() > kRoomy) {
      c->nl = 4u;
      if (bytes() <= kRoomy) c->nll = 2u;
      else c->nl = 1u << c->nll;
    }
    while (c->ng > 2u && !fits()) --c->ng;
    if (!fits()) { c->nsl = 1; c->ns = 2; }
    if (!fits()) { c->nll = 2; c->nl = 4; }
  }
  while (c->ng > 1u && !fits()) --c->ng;
  // with the small L1 the afferent cache's reads cost more than they save (us per step,
  // without / with it: 74 / 70 at 160, 89 / 86 at 256, 104 / 101 at 300; but 115 / 119 at 352
  // and 163 / 170 at 512)
  c->aff = direct || bytes() <= 195u * 1024u ? 1u : 0u;
  // a list for each of a CTA's columns, within 160 KiB (four teams of 4,096 columns, us per step
  // without / with 122 to 147 KiB of lists: 293 / 265 at 160 trajectories in the largest, 240 / 209 at 127)
  if (direct && B > 32u) {
    c->nl = cols;
    if (c->nl * list_words((B + 31u) / 32u) * 4u > 160u * 1024u || !fits()) c->nl = 0;
  }
  return bytes();
}
}  // namespace

}  // namespace axon
