// The step loop of one presentation, run by a team of CTAs that owns every column of a
// network: the whole grid in the plain kernel, a slot's CTAs in the multi-network kernel.
// See plain.cu for the phases.
#pragma once
#include <cstdint>

#include "axon_device.cuh"
#include "batch_common.cuh"
#include "emit.cuh"
#include "learn.cuh"
#include "plain.cuh"
#include "theta.cuh"

namespace axon {

// The CTAs that run a presentation together.
struct PresentTeam {
  uint32_t rank, nb;   // this CTA, CTAs of the team
  uint32_t own;        // warps per CTA that own columns; the others help with copies and learning
  uint32_t poolTiles;  // W3 tiles the CTA's pool holds
  uint32_t *bar, *hist;  // barrier counter; three drive histograms
};

// A CTA's shared memory. Every function that uses it builds the map in place.
struct PresentMap {
  uint32_t *spk0, *spk1;   // spike vectors, ping-pong
  uint32_t *act0, *act1;   // group-activity bits, ping-pong
  uint32_t* stim;          // input clamp pattern
  uint32_t* hist;          // the step's drive histogram (kHistWords)
  uint32_t* flag;          // [0] barrier flag, [1] learning-task count, [2] candidates,
                           // [3] tile-pool slots claimed, [4..7] threshold select
  uint64_t* mbar;          // one per column slot (tile pool)
  uint32_t* task;          // learning tasks: (column slot << 5) | branch
  uint32_t* bbl;           // branch-NMDA masks of the learning columns
  uint32_t *ltp, *ltd;     // per-neuron potentiation and depression counts of this step
  uint32_t* firedL;        // spike ballot of each learning column
  uint32_t* colL;          // its column index
  uint32_t* mark;          // step+1 when the slot learns this step
  uint32_t* bias;          // intrinsic bias of each owned neuron (slot * 32 + lane)
  uint32_t* mul;           // assembly multiplicity of each owned neuron
  uint32_t* ref;           // reference ball of each owned column
  uint4* pool;             // phase A's tile pool; phase B reuses its start for
  uint32_t *drv, *ball, *cand;  // the staged drives and ungated ballots of the current step, and the
                                // drives of the threshold's histogram bin (up to ncol)
};
// maxCols: columns owned by the CTA
__device__ __forceinline__ PresentMap present_map(uint32_t ncol, uint32_t incols, uint32_t maxCols, int cpw) {
  extern __shared__ __align__(16) uint32_t sm[];
  const uint32_t nactw = (((ncol / 8u + 31u) / 32u) + 3u) & ~3u;  // 16-byte multiple
  PresentMap S;
  S.spk0 = sm;
  S.spk1 = sm + ncol;
  S.act0 = sm + 2 * ncol;
  S.act1 = S.act0 + nactw;
  S.stim = S.act1 + nactw;
  S.hist = S.stim + ((incols + 3u) & ~3u);
  S.flag = S.hist + kHistWords;
  S.mbar = reinterpret_cast<uint64_t*>(S.flag + 16);
  S.task = S.flag + 16 + 2 * kMaxColSlots;
  S.bbl = S.task + maxCols * 32;
  S.ltp = S.bbl + maxCols * 32;
  S.ltd = S.ltp + maxCols * 32;
  S.firedL = S.ltd + maxCols * 32;
  S.colL = S.firedL + maxCols;
  S.mark = S.colL + maxCols;
  S.bias = S.mark + maxCols;
  S.mul = S.bias + maxCols * 32;
  S.ref = S.mul + maxCols * 32;
  S.drv = sm + present_smem_layout(ncol, incols, cpw).poolWord;
  S.pool = reinterpret_cast<uint4*>(S.drv);
  S.ball = S.drv + ncol;
  S.cand = S.ball + ncol;
  return S;
}

// The columns that each warp of a CTA owns, CPW per warp. MULTI: outputs may be absent and the
// work is counted (the plain kernel always has them all).
template <int CPW, bool MULTI>
struct PresentCta {
  uint32_t ncol, incols;
  uint32_t col[CPW], cn[CPW];
  uint32_t mph;  // bit i: phase parity of column slot i's mbarrier
  uint32_t nTiles, nTasks;  // W3 tiles this warp read, learning tasks of the CTA

  // once per launch
  __device__ __forceinline__ void init(uint32_t ncol_, uint32_t incols_, const PresentTeam& tm) {
    ncol = ncol_;
    incols = incols_;
    const PresentMap S = present_map(ncol, incols, tm.own * CPW, CPW);
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
      for (uint32_t i = 0; i < tm.own * CPW; ++i) mbar_init(&S.mbar[i], 1);
      fence_proxy_async_smem();
    }
    // columns are dealt to warps CTA-interleaved (column = warp * team + CTA): the clamped
    // input columns, which all fire and learn during the clamp, spread over every CTA instead
    // of loading the first few
    const uint32_t gwarp = warp < tm.own ? warp * tm.nb + tm.rank : ncol, nwarps = tm.nb * tm.own;
#pragma unroll
    for (int i = 0; i < CPW; ++i) col[i] = gwarp + (uint32_t)i * nwarps;
    mph = nTiles = nTasks = 0;
  }

  // once per network: the owned columns' conn rows (lane = branch) in registers, the rest of
  // their per-neuron state in shared memory by column slot (warp * CPW + i)
  __device__ __forceinline__ void load(const NetDev& d, const PresentTeam& tm) {
    const PresentMap S = present_map(ncol, incols, tm.own * CPW, CPW);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < CPW; ++i) {
      cn[i] = 0u;
      const uint32_t slot = warp * CPW + (uint32_t)i;
      if (col[i] < ncol) {
        cn[i] = d.conn[col[i] * kNslot + lane];
        S.bias[slot * 32u + lane] = d.bias[col[i] * 32u + lane];
        S.mul[slot * 32u + lane] = d.mult[col[i] * 32u + lane];
        if (!MULTI && lane == 0) S.ref[slot] = d.refBall[col[i]];
      }
    }
  }

  // once per presentation, before a block barrier
  __device__ __forceinline__ void begin(const NetDev& d, const PresentTeam& tm) {
    const PresentMap S = present_map(ncol, incols, tm.own * CPW, CPW);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    for (uint32_t i = tid; i < ncol; i += blockDim.x) S.spk0[i] = 0u;
    for (uint32_t i = tid; i < (uint32_t)(S.act1 - S.act0); i += blockDim.x) S.act0[i] = 0u;
    for (uint32_t i = tid; i < tm.own * CPW; i += blockDim.x) S.mark[i] = 0u;
    if (tid == 0) S.flag[1] = S.flag[3] = 0u;
    for (uint32_t i = tid; i < incols; i += blockDim.x) S.stim[i] = d.stim[i];
#pragma unroll
    for (int i = 0; MULTI && i < CPW; ++i)
      if (col[i] < ncol && lane == 0) S.ref[warp * CPW + (uint32_t)i] = d.refBall ? d.refBall[col[i]] : 0u;
  }

  // The T steps; g0 = steps the team has run before (barrier epoch, exchange parity and
  // histogram follow the team's step count). LEARN is c.learn as a template argument: readouts
  // carry none of the learning code's register pressure. Returns false when a grid wait gave up.
  template <bool LEARN>
  __device__ __forceinline__ bool steps(const NetDev& d, const PresentCfg& c, const PresentTeam& tm, uint32_t g0) {
    // the sizes, and the shared-memory map from them, come from the kernel's parameters instead of being held
    // for the launch: a readout step of 2,080 columns takes 6.35 us (drive 2.21, spikes 1.82) against 6.47
    // (2.25, 1.88), a 10-step learning call of 6,144 columns 252 against 260 us. Learning with one column per
    // warp is the other way round (4,096 columns: 202 against 189 us)
    const uint32_t ncol = MULTI || (LEARN && CPW == 1) ? this->ncol : c.ncol, incols = MULTI || (LEARN && CPW == 1) ? this->incols : c.incols;
    const PresentMap S = present_map(ncol, incols, tm.own * CPW, CPW);
    const uint32_t ngrp = ncol / 8u, poolTiles = tm.poolTiles;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, wpb = blockDim.x >> 5;
    // branch term of k_drive (src/axon.mm:174-178): the count (modes 0, 1) plus, when the
    // branch reaches dthr, the boost (mode 1) or 1 (mode 2)
    const uint32_t linMask = c.mode != 2u ? kFull : 0u;
    const uint32_t addN = c.mode == 1u ? c.boost : (c.mode == 2u ? 1u : 0u);

    // what phase A leaves for phase C; readout launches keep a step's values until its records
    // are written, during the next step's tile copies
    uint32_t acc[CPW], bb[CPW], vk[CPW], vk1[CPW];
#pragma unroll
    for (int i = 0; i < CPW; ++i) acc[i] = bb[i] = vk[i] = vk1[i] = 0u;
    // Records of column slot i for step tr, whose spike ballot is bw: the final state at the
    // last step, stats[2] and driveLog (src/axon.mm:213-220), hist and the k_emit counters
    // (src/axon.mm:224-234).
    auto records = [&](int i, uint32_t tr, uint32_t bw) {
      const uint32_t cc = col[i];
      const uint32_t slot = warp * CPW + (uint32_t)i;
      const bool recur = cc >= incols;
      const bool fired = (bw >> lane) & 1u;
      if (tr + 1u == c.T) {  // final state of the owned neurons, as present() leaves it
        d.acc[cc * 32u + lane] = acc[i];
        d.bbits[cc * 32u + lane] = bb[i];
        if (lane == 0) d.marg[cc] = vk[i] > vk1[i] ? 1u : 0u;
      }
      if (recur) {
        const uint32_t coinc = __reduce_add_sync(kFull, fired ? (uint32_t)__popc(bb[i]) : 0u);
        const bool member = (S.ref[slot] >> lane) & 1u;
        const bool shared = S.mul[slot * 32u + lane] > 1u;
        const uint32_t mS = __ballot_sync(kFull, member && shared), mE = __ballot_sync(kFull, member && !shared);
        const uint32_t sumS = __reduce_add_sync(kFull, (member && shared) ? acc[i] : 0u);
        const uint32_t sumE = __reduce_add_sync(kFull, (member && !shared) ? acc[i] : 0u);
        if (lane == 0) {
          if (coinc && (!MULTI || d.stats)) atomicAdd(d.stats + 2, coinc);
          if (mS) { atomicAdd(d.driveLog + tr * 4u + 0u, sumS); atomicAdd(d.driveLog + tr * 4u + 1u, (uint32_t)__popc(mS)); }
          if (mE) { atomicAdd(d.driveLog + tr * 4u + 2u, sumE); atomicAdd(d.driveLog + tr * 4u + 3u, (uint32_t)__popc(mE)); }
        }
      }
      if (lane == 0) {
        if (!MULTI || d.hist) d.hist[(size_t)tr * ncol + cc] = bw;
        if (bw != 0u && recur && (!MULTI || d.stats)) {
          const uint32_t sb = 64u + tr * 8u;
          atomicAdd(d.stats + 0, 1u);
          atomicAdd(d.stats + 1, (uint32_t)__popc(bw));
          atomicAdd(d.stats + sb + 0u, vk[i] - vk1[i]);
          atomicAdd(d.stats + sb + 1u, vk[i]);
          atomicAdd(d.stats + sb + 2u, 1u);
          if (vk[i] == vk1[i]) atomicAdd(d.stats + sb + 3u, 1u);
          if (vk[i] == 0u) atomicAdd(d.stats + sb + 4u, 1u);
        }
      }
    };

    for (uint32_t t = 0; t < c.T; ++t) {
      const uint32_t* sIn = (t & 1u) ? S.spk1 : S.spk0;
      uint32_t* sOut = (t & 1u) ? S.spk0 : S.spk1;
      const uint32_t* sActIn = (t & 1u) ? S.act1 : S.act0;
      uint32_t* sActOut = (t & 1u) ? S.act0 : S.act1;
      const uint4* sIn4 = reinterpret_cast<const uint4*>(sIn);
      const uint32_t g = g0 + t, par = g & 1u, h3 = g % 3u;
      const bool clamp = t < c.clampSteps;
      const uint32_t phase = (!LEARN || !c.contrast) ? 0u
                             : (clamp ? 1u : (((t - c.clampSteps) % c.ltdEvery == 0u) ? 2u : 3u));
      if (LEARN) {
#pragma unroll
        for (int i = 0; i < CPW; ++i) acc[i] = bb[i] = vk[i] = vk1[i] = 0u;
      }

      // per-phase device timer stamps of the profile mode (thread 0 of every CTA)
      unsigned long long* stamp = d.prof ? d.prof + ((size_t)t * tm.nb + tm.rank) * 5u : nullptr;
      if (stamp && tid == 0) stamp[0] = globaltimer_ns();
      // ---------------- phase A: drive (k_drive, src/axon.mm:150-190) + ungated k-WTA
      // The owner warp claims one pool slot per non-silent branch of its column; the lane of
      // each such branch issues the tile's bulk copy, so all of the CTA's tiles are in flight
      // together. A column whose claim does not fit the pool streams its tiles through
      // registers instead, four at a time. Spikes come from shared memory.
#pragma unroll
      for (int i = 0; i < CPW; ++i) {
        if (col[i] >= ncol) continue;  // warp-uniform
        const uint32_t cc = col[i];
        const bool on = (sActIn[cn[i] >> 5] >> (cn[i] & 31u)) & 1u;
        uint32_t active = __ballot_sync(kFull, on);
        const uint32_t n = (uint32_t)__popc(active);
        if (MULTI) nTiles += n;
        uint32_t a = 0, b2 = 0;
        uint32_t slot0 = 0;
        if (lane == 0 && n != 0u) slot0 = atomicAdd(S.flag + 3, n);
        slot0 = __shfl_sync(kFull, slot0, 0);
        const bool pooled = n != 0u && slot0 + n <= poolTiles;
        uint64_t* mb = &S.mbar[warp * CPW + (uint32_t)i];
        if (pooled) {
          if (lane == 0) mbar_expect_tx(mb, n * 1024u);
          __syncwarp();
          if (on) {
            const uint32_t r = (uint32_t)__popc(active & ((1u << lane) - 1u));
            if (LEARN) fence_proxy_async_all();
            else fence_proxy_async_smem();
            bulk_g2s(S.pool + (size_t)(slot0 + r) * kTileU4, d.W3 + ((size_t)cc * kNslot + lane) * kTileU4, 1024u, mb);
          }
        }
        // a readout writes the previous step's records while this step's tiles are in flight
        if (!LEARN) {
          if (t > 0u) records(i, t - 1u, sIn[cc]);
          acc[i] = bb[i] = vk[i] = vk1[i] = 0u;
        }
        if (pooled) {
          const uint32_t ph = (mph >> i) & 1u;
          if (!mbar_wait(mb, ph, c.waitNs)) {
            // the copies did not land in time: record it, wait (bounded) for them, and let
            // the grid barrier end the launch
            if (lane == 0) atomicCAS(d.err, 0u, kErrTimeout);
            mbar_wait(mb, ph, c.waitNs > kDrainNs ? c.waitNs : kDrainNs);
          }
          mph ^= 1u << i;
          const uint4* T = S.pool + (size_t)slot0 * kTileU4 + lane;
          for (uint32_t r = 0; active; ++r, T += kTileU4) {
            const uint32_t s = (uint32_t)(__ffs(active) - 1);
            active &= active - 1u;
            const uint32_t g = __shfl_sync(kFull, cn[i], s);
            const uint32_t cnt = popc4(T[0], sIn4[2 * g]) + popc4(T[32], sIn4[2 * g + 1]);
            const bool nmda = cnt >= c.dthr;
            if (nmda) b2 |= 1u << s;
            a += (cnt & linMask) + (nmda ? addN : 0u);
          }
        } else {
          const uint4* Wt = d.W3 + (size_t)cc * kNslot * kTileU4 + lane;
          while (active) {
            uint32_t s[4];
            bool v[4];
            uint4 w0[4], w1[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              v[u] = active != 0u;
              s[u] = v[u] ? (uint32_t)(__ffs(active) - 1) : 0u;
              active &= active - 1u;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (v[u]) {
                w0[u] = __ldcg(Wt + s[u] * kTileU4);
                w1[u] = __ldcg(Wt + s[u] * kTileU4 + 32);
              }
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (v[u]) {
                const uint32_t g = __shfl_sync(kFull, cn[i], s[u]);
                const uint32_t cnt = popc4(w0[u], sIn4[2 * g]) + popc4(w1[u], sIn4[2 * g + 1]);
                const bool nmda = cnt >= c.dthr;
                if (nmda) b2 |= 1u << s[u];
                a += (cnt & linMask) + (nmda ? addN : 0u);
              }
          }
        }
        if (c.facil != 0u && ((sIn[cc] >> lane) & 1u)) a += c.facil;
        const uint32_t bi = c.useBias ? (S.bias[(warp * CPW + (uint32_t)i) * 32u + lane] >> c.biasShift) : 0u;
        a = a > bi ? a - bi : 0u;
        acc[i] = a;
        bb[i] = b2;
        const uint32_t drv = __reduce_add_sync(kFull, a);
        const uint32_t ball = warp_kwta(a, lane, c.k, vk[i], vk1[i]);
        if (lane == 0) {
          __stcg(d.xdrive + par * ncol + cc, drv);
          __stcg(d.xball + par * ncol + cc, ball);
          if (cc >= incols && drv < (1u << 24)) {
            uint32_t* h = tm.hist + h3 * kHistWords + theta_key(drv);
            atomicAdd(h, 1u);
            atomicMax(h + kThetaBins, drv);
            atomicMax(h + 2u * kThetaBins, ~drv);
          }
          if (t + 1u == c.T) d.drive[cc] = drv;  // final state: the last step's column drive
        }
      }

      if (stamp) {
        __syncthreads();
        if (tid == 0) stamp[1] = globaltimer_ns();
      }
      if (!grid_barrier(tm.bar, d.err, tm.nb + c.missing, g0 + t, c.waitNs, S.flag)) return false;
      if (stamp && tid == 0) stamp[2] = globaltimer_ns();

      // ---------------- phase B: column threshold (k_topk) and the full spike vector
      // this step's drive histogram, the drives and the ballots come from L2 by asynchronous
      // copies, in that order (three groups): warp 0 scans the histogram while the drives and
      // ballots keep arriving
      for (uint32_t i = tid; i < kHistWords / 4u; i += blockDim.x)
        cp_async16(reinterpret_cast<uint4*>(S.hist) + i, reinterpret_cast<const uint4*>(tm.hist + h3 * kHistWords) + i);
      cp_async_commit();
      for (uint32_t i = tid; i < ncol / 4u; i += blockDim.x)
        cp_async16(reinterpret_cast<uint4*>(S.drv) + i, reinterpret_cast<const uint4*>(d.xdrive + par * ncol) + i);
      cp_async_commit();
      for (uint32_t i = tid; i < ncol / 4u; i += blockDim.x)
        cp_async16(reinterpret_cast<uint4*>(S.ball) + i, reinterpret_cast<const uint4*>(d.xball + par * ncol) + i);
      cp_async_commit();
      if (tid == 0) { S.flag[2] = 0u; S.flag[3] = 0u; }  // every warp has claimed its pool slots
      // histogram g+2 (last read in step g-1, before this barrier) is cleared for its next use
      if (tm.rank == 0 && g >= 1u)
        for (uint32_t i = tid; i < kHistWords; i += blockDim.x) __stcg(tm.hist + ((g + 2u) % 3u) * kHistWords + i, 0u);
      cp_async_wait<2>();  // the histogram
      __syncthreads();
      const uint32_t theta = hist_theta<1>(S.drv, S.hist, S.cand, S.flag + 2, incols, ncol, c.targetCols, c.topkPar);
      const uint32_t gate = max(theta, 1u);
      cp_async_wait<0>();
      __syncthreads();
      emit_groups(S.drv, S.ball, S.stim, sOut, sActOut, gate, clamp, incols, ngrp);
      __syncthreads();
      if (tm.rank == 0 && tid == 0) { d.theta[0] = theta; d.theta[1] = 0u; }

      if (stamp && tid == 0) stamp[3] = globaltimer_ns();
      // ---------------- phase C: own-column records, bias and learning
#pragma unroll
      for (int i = 0; i < CPW; ++i) {
        if (col[i] >= ncol) continue;
        const uint32_t cc = col[i];
        const uint32_t slot = warp * CPW + (uint32_t)i;
        const uint32_t b = sOut[cc];
        const bool recur = cc >= incols;
        const bool fired = (b >> lane) & 1u;
        if (!LEARN) continue;  // a readout's records wait for the next step's tile copies
        records(i, t, b);
        // k_bias, src/axon.mm:240-253
        if (recur) {
          const int dec = ((t % max(c.biasDownEvery, 1u)) == 0u) ? (int)c.biasDown : 0;
          const int nb = (int)S.bias[slot * 32u + lane] + (fired ? (int)c.biasUp : -dec);
          S.bias[slot * 32u + lane] = (uint32_t)max(0, nb);
        }
        // k_learn, src/axon.mm:436-495: each voted branch of a learning column becomes a
        // task that any warp of the CTA runs, so a column's read-modify-writes overlap
        if (phase == 3u || b == 0u) continue;
        if (c.marginGate != 0u && !(vk[i] > vk1[i])) continue;
        const uint32_t vmask = __reduce_or_sync(kFull, fired ? bb[i] : 0u);
        S.bbl[slot * 32u + lane] = bb[i];
        S.ltp[slot * 32u + lane] = 0u;
        S.ltd[slot * 32u + lane] = 0u;
        if (lane == 0) { S.firedL[slot] = b; S.colL[slot] = cc; S.mark[slot] = t + 1u; }
        if ((vmask >> lane) & 1u) S.task[atomicAdd(S.flag + 1, 1u)] = (slot << 5) | lane;
      }
      if (LEARN) {
        __syncthreads();
        const uint32_t ntask = S.flag[1];
        if (MULTI) nTasks += ntask;
        for (uint32_t k = warp; k < ntask; k += wpb) {
          const uint32_t tk = S.task[k], slot = tk >> 5, s = tk & 31u;
          const uint32_t cc = S.colL[slot];
          const bool want = ((S.firedL[slot] >> lane) & 1u) && ((S.bbl[slot * 32u + lane] >> s) & 1u);
          const uint32_t g = __ldg(d.conn + cc * kNslot + s);
          const size_t base = ((size_t)cc * kNslot + s) * kTileU4 + lane;
          uint4 p0[2], p1[2], p2[2], p3[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            p0[j] = __ldcg(d.W0 + base + 32 * j);
            p1[j] = __ldcg(d.W1 + base + 32 * j);
            p2[j] = __ldcg(d.W2 + base + 32 * j);
            p3[j] = __ldcg(d.W3 + base + 32 * j);
          }
          const Band band = band_of(c.bandLo, c.bandHi);
          uint32_t nLTP = 0, nLTD = 0;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint4 sp4 = sIn4[2 * g + j];
            learn_word(p0[j].x, p1[j].x, p2[j].x, p3[j].x, sp4.x, want, phase, t, c, band, nLTP, nLTD);
            learn_word(p0[j].y, p1[j].y, p2[j].y, p3[j].y, sp4.y, want, phase, t, c, band, nLTP, nLTD);
            learn_word(p0[j].z, p1[j].z, p2[j].z, p3[j].z, sp4.z, want, phase, t, c, band, nLTP, nLTD);
            learn_word(p0[j].w, p1[j].w, p2[j].w, p3[j].w, sp4.w, want, phase, t, c, band, nLTP, nLTD);
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            __stcg(d.W0 + base + 32 * j, p0[j]);
            __stcg(d.W1 + base + 32 * j, p1[j]);
            __stcg(d.W2 + base + 32 * j, p2[j]);
            __stcg(d.W3 + base + 32 * j, p3[j]);
          }
          fence_proxy_async_all();  // the next step copies W3 tiles in bulk (async proxy)
          if (nLTP) atomicAdd(S.ltp + slot * 32u + lane, nLTP);
          if (nLTD) atomicAdd(S.ltd + slot * 32u + lane, nLTD);
        }
        __syncthreads();
        // plasticity counters per neuron and step, src/axon.mm:491-494
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
          const uint32_t slot = warp * CPW + (uint32_t)i;
          if (col[i] >= ncol || S.mark[slot] != t + 1u) continue;  // (helper warps own no column)
          const uint32_t nLTP = S.ltp[slot * 32u + lane], nLTD = S.ltd[slot * 32u + lane];
          const uint32_t sumP = __reduce_add_sync(kFull, nLTP), sumD = __reduce_add_sync(kFull, nLTD);
          const uint32_t kP = __popc(__ballot_sync(kFull, nLTP != 0u)), kD = __popc(__ballot_sync(kFull, nLTD != 0u));
          if (lane == 0 && (!MULTI || d.stats)) {
            if (sumP) atomicAdd(d.stats + 8, sumP);
            if (sumD) atomicAdd(d.stats + 9, sumD);
            if (kP) atomicAdd(d.stats + 10, kP);
            if (kD) atomicAdd(d.stats + 11, kD);
          }
        }
        if (tid == 0) S.flag[1] = 0u;
      }
      __syncthreads();  // sOut / sActOut complete before the next step reads them
      if (stamp && tid == 0) stamp[4] = globaltimer_ns();
    }

    if (!LEARN) {  // the last step's records
      const uint32_t* sLast = (c.T & 1u) ? S.spk1 : S.spk0;
#pragma unroll
      for (int i = 0; i < CPW; ++i)
        if (col[i] < ncol) records(i, c.T - 1u, sLast[col[i]]);
    }
    return true;
  }

  // final state of a presentation, as the reference's buffers hold it after present()
  __device__ __forceinline__ void end(const NetDev& d, const PresentTeam& tm, uint32_t T) {
    const PresentMap S = present_map(ncol, incols, tm.own * CPW, CPW);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t* sLast = (T & 1u) ? S.spk1 : S.spk0;   // spk(T-1)
    const uint32_t* sPrev = (T & 1u) ? S.spk0 : S.spk1;   // spk(T-2), zero when T == 1
    uint32_t* gLast = ((T - 1u) & 1u) ? d.spkA : d.spkB;
    uint32_t* gPrev = ((T - 1u) & 1u) ? d.spkB : d.spkA;
#pragma unroll
    for (int i = 0; i < CPW; ++i) {
      if (col[i] >= ncol || lane != 0u) continue;
      const uint32_t cc = col[i];
      gLast[cc] = sLast[cc];
      gPrev[cc] = T >= 2u ? sPrev[cc] : 0u;
      if (d.finalOut) d.finalOut[cc] = sLast[cc];
    }
  }

  // the biases that learning changed
  __device__ __forceinline__ void store_bias(const NetDev& d, const PresentTeam& tm) {
    const PresentMap S = present_map(ncol, incols, tm.own * CPW, CPW);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < CPW; ++i)
      if (col[i] < ncol) d.bias[col[i] * 32u + lane] = S.bias[(warp * CPW + (uint32_t)i) * 32u + lane];
  }
};

}  // namespace axon
