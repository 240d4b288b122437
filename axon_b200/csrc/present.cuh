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

// A CTA's shared memory and the columns each of its warps owns, CPW per warp.
template <int CPW>
struct PresentCta {
  uint32_t *sSpk0, *sSpk1, *sAct0, *sAct1, *sStim, *sHist, *sFlag, *sTask, *sBBL, *sLTP, *sLTD, *sFiredL, *sColL, *sMark,
      *sBias, *sMul, *sRef, *sD, *sB, *sCand;
  uint64_t* sMbar;
  uint4* sPool;
  uint32_t ncol, incols, nactw, maxCols;
  uint32_t col[CPW], cn[CPW];
  uint32_t mph;  // bit i: phase parity of column slot i's mbarrier
  uint32_t nTiles, nTasks;  // W3 tiles this warp read, learning tasks of the CTA

  // once per launch
  __device__ __forceinline__ void init(uint32_t* sm, uint32_t ncol_, uint32_t incols_, const PresentTeam& tm) {
    ncol = ncol_;
    incols = incols_;
    const uint32_t ngrp = ncol / 8u, tid = threadIdx.x, warp = tid >> 5;
    nactw = (((ngrp + 31u) / 32u) + 3u) & ~3u;  // 16-byte multiple
    maxCols = tm.own * CPW;                     // columns owned by this CTA
    const PresentSmem L = present_smem_layout(ncol, incols, CPW);
    sSpk0 = sm;                    // spike vectors, ping-pong
    sSpk1 = sm + ncol;
    sAct0 = sm + 2 * ncol;         // group-activity bits, ping-pong
    sAct1 = sAct0 + nactw;
    sStim = sAct1 + nactw;         // input clamp pattern
    sHist = sStim + ((incols + 3u) & ~3u);  // the step's drive histogram (kHistWords)
    sFlag = sHist + kHistWords;    // [0] barrier flag, [1] learning-task count, [2] candidates,
                                   // [3] tile-pool slots claimed, [4..7] threshold select
    sMbar = reinterpret_cast<uint64_t*>(sFlag + 16);  // one per column slot (tile pool)
    sTask = sFlag + 16 + 2 * kMaxColSlots;  // learning tasks: (column slot << 5) | branch
    sBBL = sTask + maxCols * 32;   // branch-NMDA masks of the learning columns
    sLTP = sBBL + maxCols * 32;    // per-neuron potentiation counts of this step
    sLTD = sLTP + maxCols * 32;    // per-neuron depression counts
    sFiredL = sLTD + maxCols * 32; // spike ballot of each learning column
    sColL = sFiredL + maxCols;     // its column index
    sMark = sColL + maxCols;       // step+1 when the slot learns this step
    sBias = sMark + maxCols;       // intrinsic bias of each owned neuron (slot * 32 + lane)
    sMul = sBias + maxCols * 32;   // assembly multiplicity of each owned neuron
    sRef = sMul + maxCols * 32;    // reference ball of each owned column
    // phase A's tile pool; phase B reuses its start for the staged drives, the ungated
    // ballots and the threshold candidates
    sPool = reinterpret_cast<uint4*>(sm + L.poolWord);
    sD = sm + L.poolWord;          // staged drives of the current step
    sB = sD + ncol;                // staged ungated ballots
    sCand = sB + ncol;             // drives of the threshold's histogram bin (up to ncol)
    if (tid == 0) {
      for (uint32_t i = 0; i < maxCols; ++i) mbar_init(&sMbar[i], 1);
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
  __device__ __forceinline__ void load(const NetDev& d) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < CPW; ++i) {
      cn[i] = 0u;
      const uint32_t slot = warp * CPW + (uint32_t)i;
      if (col[i] < ncol) {
        cn[i] = d.conn[col[i] * kNslot + lane];
        sBias[slot * 32u + lane] = d.bias[col[i] * 32u + lane];
        sMul[slot * 32u + lane] = d.mult[col[i] * 32u + lane];
      }
    }
  }

  // once per presentation, before a block barrier
  __device__ __forceinline__ void begin(const NetDev& d) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    for (uint32_t i = tid; i < ncol; i += blockDim.x) sSpk0[i] = 0u;
    for (uint32_t i = tid; i < nactw; i += blockDim.x) sAct0[i] = 0u;
    for (uint32_t i = tid; i < maxCols; i += blockDim.x) sMark[i] = 0u;
    if (tid == 0) sFlag[1] = sFlag[3] = 0u;
    for (uint32_t i = tid; i < incols; i += blockDim.x) sStim[i] = d.stim[i];
#pragma unroll
    for (int i = 0; i < CPW; ++i)
      if (col[i] < ncol && lane == 0) sRef[warp * CPW + (uint32_t)i] = d.refBall ? d.refBall[col[i]] : 0u;
  }

  // The T steps; g0 = steps the team has run before (barrier epoch, exchange parity and
  // histogram follow the team's step count). LEARN is c.learn as a template argument: readouts
  // carry none of the learning code's register pressure. Returns false when a grid wait gave up.
  template <bool LEARN>
  __device__ __forceinline__ bool steps(const NetDev& d, const PresentCfg& c, const PresentTeam& tm, uint32_t g0) {
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
        const bool member = (sRef[slot] >> lane) & 1u;
        const bool shared = sMul[slot * 32u + lane] > 1u;
        const uint32_t mS = __ballot_sync(kFull, member && shared), mE = __ballot_sync(kFull, member && !shared);
        const uint32_t sumS = __reduce_add_sync(kFull, (member && shared) ? acc[i] : 0u);
        const uint32_t sumE = __reduce_add_sync(kFull, (member && !shared) ? acc[i] : 0u);
        if (lane == 0) {
          if (coinc && d.stats) atomicAdd(d.stats + 2, coinc);
          if (mS) { atomicAdd(d.driveLog + tr * 4u + 0u, sumS); atomicAdd(d.driveLog + tr * 4u + 1u, (uint32_t)__popc(mS)); }
          if (mE) { atomicAdd(d.driveLog + tr * 4u + 2u, sumE); atomicAdd(d.driveLog + tr * 4u + 3u, (uint32_t)__popc(mE)); }
        }
      }
      if (lane == 0) {
        if (d.hist) d.hist[(size_t)tr * ncol + cc] = bw;
        if (bw != 0u && recur && d.stats) {
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
      const uint32_t* sIn = (t & 1u) ? sSpk1 : sSpk0;
      uint32_t* sOut = (t & 1u) ? sSpk0 : sSpk1;
      const uint32_t* sActIn = (t & 1u) ? sAct1 : sAct0;
      uint32_t* sActOut = (t & 1u) ? sAct0 : sAct1;
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
        nTiles += n;
        uint32_t a = 0, b2 = 0;
        uint32_t slot0 = 0;
        if (lane == 0 && n != 0u) slot0 = atomicAdd(sFlag + 3, n);
        slot0 = __shfl_sync(kFull, slot0, 0);
        const bool pooled = n != 0u && slot0 + n <= poolTiles;
        uint64_t* mb = &sMbar[warp * CPW + (uint32_t)i];
        if (pooled) {
          if (lane == 0) mbar_expect_tx(mb, n * 1024u);
          __syncwarp();
          if (on) {
            const uint32_t r = (uint32_t)__popc(active & ((1u << lane) - 1u));
            if (LEARN) fence_proxy_async_all();
            else fence_proxy_async_smem();
            bulk_g2s(sPool + (size_t)(slot0 + r) * kTileU4, d.W3 + ((size_t)cc * kNslot + lane) * kTileU4, 1024u, mb);
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
          const uint4* T = sPool + (size_t)slot0 * kTileU4 + lane;
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
        const uint32_t bi = c.useBias ? (sBias[(warp * CPW + (uint32_t)i) * 32u + lane] >> c.biasShift) : 0u;
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
      if (!grid_barrier(tm.bar, d.err, tm.nb + c.missing, g0 + t, c.waitNs, sFlag)) return false;
      if (stamp && tid == 0) stamp[2] = globaltimer_ns();

      // ---------------- phase B: column threshold (k_topk) and the full spike vector
      // this step's drive histogram, the drives and the ballots come from L2 by asynchronous
      // copies, in that order (three groups): warp 0 scans the histogram while the drives and
      // ballots keep arriving
      for (uint32_t i = tid; i < kHistWords / 4u; i += blockDim.x)
        cp_async16(reinterpret_cast<uint4*>(sHist) + i, reinterpret_cast<const uint4*>(tm.hist + h3 * kHistWords) + i);
      cp_async_commit();
      for (uint32_t i = tid; i < ncol / 4u; i += blockDim.x)
        cp_async16(reinterpret_cast<uint4*>(sD) + i, reinterpret_cast<const uint4*>(d.xdrive + par * ncol) + i);
      cp_async_commit();
      for (uint32_t i = tid; i < ncol / 4u; i += blockDim.x)
        cp_async16(reinterpret_cast<uint4*>(sB) + i, reinterpret_cast<const uint4*>(d.xball + par * ncol) + i);
      cp_async_commit();
      if (tid == 0) { sFlag[2] = 0u; sFlag[3] = 0u; }  // every warp has claimed its pool slots
      // histogram g+2 (last read in step g-1, before this barrier) is cleared for its next use
      if (tm.rank == 0 && g >= 1u)
        for (uint32_t i = tid; i < kHistWords; i += blockDim.x) __stcg(tm.hist + ((g + 2u) % 3u) * kHistWords + i, 0u);
      cp_async_wait<2>();  // the histogram
      __syncthreads();
      const uint32_t theta = hist_theta<1>(sD, sHist, sCand, sFlag + 2, incols, ncol, c.targetCols, c.topkPar);
      const uint32_t gate = max(theta, 1u);
      cp_async_wait<0>();
      __syncthreads();
      emit_groups(sD, sB, sStim, sOut, sActOut, gate, clamp, incols, ngrp);
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
          const int nb = (int)sBias[slot * 32u + lane] + (fired ? (int)c.biasUp : -dec);
          sBias[slot * 32u + lane] = (uint32_t)max(0, nb);
        }
        // k_learn, src/axon.mm:436-495: each voted branch of a learning column becomes a
        // task that any warp of the CTA runs, so a column's read-modify-writes overlap
        if (phase == 3u || b == 0u) continue;
        if (c.marginGate != 0u && !(vk[i] > vk1[i])) continue;
        const uint32_t vmask = __reduce_or_sync(kFull, fired ? bb[i] : 0u);
        sBBL[slot * 32u + lane] = bb[i];
        sLTP[slot * 32u + lane] = 0u;
        sLTD[slot * 32u + lane] = 0u;
        if (lane == 0) { sFiredL[slot] = b; sColL[slot] = cc; sMark[slot] = t + 1u; }
        if ((vmask >> lane) & 1u) sTask[atomicAdd(sFlag + 1, 1u)] = (slot << 5) | lane;
      }
      if (LEARN) {
        __syncthreads();
        const uint32_t ntask = sFlag[1];
        nTasks += ntask;
        for (uint32_t k = warp; k < ntask; k += wpb) {
          const uint32_t tk = sTask[k], slot = tk >> 5, s = tk & 31u;
          const uint32_t cc = sColL[slot];
          const bool want = ((sFiredL[slot] >> lane) & 1u) && ((sBBL[slot * 32u + lane] >> s) & 1u);
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
          if (nLTP) atomicAdd(sLTP + slot * 32u + lane, nLTP);
          if (nLTD) atomicAdd(sLTD + slot * 32u + lane, nLTD);
        }
        __syncthreads();
        // plasticity counters per neuron and step, src/axon.mm:491-494
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
          const uint32_t slot = warp * CPW + (uint32_t)i;
          if (col[i] >= ncol || sMark[slot] != t + 1u) continue;  // (helper warps own no column)
          const uint32_t nLTP = sLTP[slot * 32u + lane], nLTD = sLTD[slot * 32u + lane];
          const uint32_t sumP = __reduce_add_sync(kFull, nLTP), sumD = __reduce_add_sync(kFull, nLTD);
          const uint32_t kP = __popc(__ballot_sync(kFull, nLTP != 0u)), kD = __popc(__ballot_sync(kFull, nLTD != 0u));
          if (lane == 0 && d.stats) {
            if (sumP) atomicAdd(d.stats + 8, sumP);
            if (sumD) atomicAdd(d.stats + 9, sumD);
            if (kP) atomicAdd(d.stats + 10, kP);
            if (kD) atomicAdd(d.stats + 11, kD);
          }
        }
        if (tid == 0) sFlag[1] = 0u;
      }
      __syncthreads();  // sOut / sActOut complete before the next step reads them
      if (stamp && tid == 0) stamp[4] = globaltimer_ns();
    }

    if (!LEARN) {  // the last step's records
      const uint32_t* sLast = (c.T & 1u) ? sSpk1 : sSpk0;
#pragma unroll
      for (int i = 0; i < CPW; ++i)
        if (col[i] < ncol) records(i, c.T - 1u, sLast[col[i]]);
    }
    return true;
  }

  // final state of a presentation, as the reference's buffers hold it after present()
  __device__ __forceinline__ void end(const NetDev& d, uint32_t T) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t* sLast = (T & 1u) ? sSpk1 : sSpk0;   // spk(T-1)
    const uint32_t* sPrev = (T & 1u) ? sSpk0 : sSpk1;   // spk(T-2), zero when T == 1
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
  __device__ __forceinline__ void store_bias(const NetDev& d) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < CPW; ++i)
      if (col[i] < ncol) d.bias[col[i] * 32u + lane] = sBias[(warp * CPW + (uint32_t)i) * 32u + lane];
  }
};

}  // namespace axon
