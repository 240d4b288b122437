// Plain AXON path on sm_100a: one persistent launch runs all T steps of a presentation.
//
// Reference: rakib-nyc/axon src/axon.mm. There, present() (src/axon.mm:815-888) encodes
// T x {k_drive, k_topk, k_emit, k_bias, k_learn} as five Metal dispatches per step. Here
// the whole step loop is one cooperative launch with ONE grid barrier per step:
//
//   phase A  each warp owns one column (lane = neuron): drive over the column's non-silent
//            branches, the exact k-of-32 ballot, and the column drive; drive + ungated
//            ballot are published, and the drive is counted into the step's histogram.
//            The W3 tiles of the non-silent branches of all the CTA's columns are in flight
//            at once: each branch's lane issues one 1 KiB TMA bulk copy into a CTA-wide
//            shared-memory pool (slots claimed per column), completed on a per-column
//            mbarrier; spikes come from shared memory.
//   barrier
//   phase B  every CTA reads all published drives/ballots (L2), selects the column
//            threshold (the target-th largest recurrent drive) and rebuilds the whole
//            spike vector spk(t) in its own shared memory; no second barrier is needed.
//   phase C  each warp finishes its own column: hist/stats/driveLog records, intrinsic
//            bias and bit-serial learning on W0..W3.
//
// Per-neuron state that only its owner touches stays on the SM for the whole presentation
// (the connection row in registers; bias and multiplicity in shared memory); HBM traffic
// per step is the W3 tiles of non-silent branches plus the learning read-modify-writes.
// The step loop is in present.cuh, which the multi-network launch shares.
#include <cstdint>

#include "axon_device.cuh"
#include "batch_common.cuh"
#include "learn.cuh"
#include "plain.cuh"
#include "present.cuh"

namespace axon {

template <int CPW, bool LEARN>
__global__ void __launch_bounds__(kPresentMaxWarps * 32, 1) k_present(NetDev d, PresentCfg c) {
  const PresentTeam tm{blockIdx.x, gridDim.x, LEARN ? c.ownWarps : blockDim.x >> 5, present_smem_layout(c.ncol, c.incols, CPW).poolTiles, d.bar,
                       d.bar + 64};
  PresentCta<CPW, false> w;
  w.init(c.ncol, c.incols, tm);
  w.begin(d, tm);
  w.load(d, tm);
  __syncthreads();
  if (!w.template steps<LEARN>(d, c, tm, 0u)) return;
  w.end(d, tm, c.T);
  if (LEARN) w.store_bias(d, tm);
}

// ---------------------------------------------------------------- launch helpers
size_t present_smem_bytes(uint32_t ncol, uint32_t incols, int cpw) {
  return present_smem_layout(ncol, incols, cpw).bytes;
}

static const void* present_fn(int cpw, bool learn) {
  switch (cpw) {
    case 1: return learn ? (const void*)k_present<1, true> : (const void*)k_present<1, false>;
    case 2: return learn ? (const void*)k_present<2, true> : (const void*)k_present<2, false>;
    default: return nullptr;
  }
}

cudaError_t launch_present(const NetDev& d, const PresentCfg& cfg, const LaunchShape& ls, cudaStream_t st) {
  PresentCfg c = cfg;
  c.ownWarps = (uint32_t)ls.wpb;
  // Learning takes a full CTA: a firing column's voted branches (up to 32 updates of 8 KiB)
  // run one per warp at a time, and the CTAs with most of them hold up the grid barrier.
  // With the owners alone (2 warps a CTA at 256 columns, 7 at 1,024, 15 at 2,080) a 10-step
  // presentation took 170 / 121 / 131 us, with full CTAs 108 / 108 / 125.
  const int warps = c.learn ? (int)kPresentMaxWarps : ls.wpb;
  void* args[] = {(void*)&d, (void*)&c};
  const void* fn = present_fn(ls.cpw, c.learn != 0u);
  if (!fn) return cudaErrorInvalidValue;
  // barrier counter and the three drive histograms start at zero
  const cudaError_t e = cudaMemsetAsync(d.bar, 0, kBarRegionWords * 4u, st);
  if (e != cudaSuccess) return e;
  return cudaLaunchCooperativeKernel(fn, dim3(ls.grid), dim3(warps * 32), args, ls.smem, st);
}

// Sets the shared-memory size of both forms (learning, readout) and returns the smaller
// number of co-resident blocks per SM.
cudaError_t present_max_blocks_per_sm(int cpw, int threads, size_t smem, int* out) {
  *out = 0;
  int best = 1 << 30;
  for (bool learn : {false, true}) {
    const void* fn = present_fn(cpw, learn);
    if (!fn) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, threads, smem);
    if (e != cudaSuccess) return e;
    best = n < best ? n : best;
  }
  *out = best;
  return cudaSuccess;
}

// ---------------------------------------------------------------- init kernels
// k_init_w, src/axon.mm:86-104: one thread per uint4 of each plane.
__global__ void k_init_w(uint4* W0, uint4* W1, uint4* W2, uint4* W3, uint32_t nAnd, uint32_t seed, uint64_t nU4) {
  const uint64_t gg = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gg >= nU4) return;
  const uint32_t g = (uint32_t)gg ^ (seed * 0x9E3779B9u);
  uint32_t m0 = kFull, m1 = kFull, m2 = kFull, m3 = kFull;
  for (uint32_t i = 0; i < nAnd; ++i) {
    m0 &= hash32(g * 32u + i * 4u + 0u);
    m1 &= hash32(g * 32u + i * 4u + 1u);
    m2 &= hash32(g * 32u + i * 4u + 2u);
    m3 &= hash32(g * 32u + i * 4u + 3u);
  }
  const uint4 m = make_uint4(m0, m1, m2, m3);
  const uint4 cc = make_uint4(hash32(g * 8u + 11u), hash32(g * 8u + 13u), hash32(g * 8u + 17u), hash32(g * 8u + 19u));
  W3[gg] = m;
  W2[gg] = make_uint4(~m.x | cc.x, ~m.y | cc.y, ~m.z | cc.z, ~m.w | cc.w);
  W1[gg] = cc;
  W0[gg] = make_uint4(~cc.x, ~cc.y, ~cc.z, ~cc.w);
}
// k_init_conn, src/axon.mm:109-117
__global__ void k_init_conn(uint32_t* conn, uint32_t nGrp, uint32_t nInGrp, uint32_t inBr, uint32_t seed, uint32_t n) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  const uint32_t s = g % kNslot;
  const uint32_t h = hash32(g * 2246822519u + 7u + seed * 2654435761u);
  conn[g] = (s < inBr) ? (h % nInGrp) : (nInGrp + h % (nGrp - nInGrp));
}

cudaError_t launch_init(const NetDev& d, uint32_t ncol, uint32_t incols, uint32_t inbr, uint32_t nand, uint32_t seed,
                        cudaStream_t st) {
  const uint64_t nU4 = (uint64_t)ncol * kNslot * kTileU4;
  k_init_w<<<(unsigned)((nU4 + 255) / 256), 256, 0, st>>>(d.W0, d.W1, d.W2, d.W3, nand, seed, nU4);
  const uint32_t n = ncol * kNslot;
  k_init_conn<<<(n + 255) / 256, 256, 0, st>>>(d.conn, ncol / 8u, incols / 8u, inbr, seed, n);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- diagnostics
// k_wstat, src/axon.mm:641-646
__global__ void k_wstat(const uint4* W3, uint64_t nU4, uint32_t* out) {
  uint32_t s = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nU4; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint4 w = __ldcs(W3 + i);
    s += __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
  }
  s = __reduce_add_sync(kFull, s);
  if ((threadIdx.x & 31u) == 0u) atomicAdd(out, s);
}

// k_within, src/axon.mm:524-562: warp per column, lane per postsynaptic neuron.
__global__ void k_within(const uint4* W3, const uint32_t* conn, const uint32_t* ball, uint32_t inBr, uint32_t inCols,
                         uint32_t ncol, uint32_t useMask, const uint32_t* postMask, const uint32_t* mult, uint32_t* out) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t colw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (colw >= ncol || colw < inCols) return;
  const uint32_t gid = colw * 32u + lane;
  bool sel = useMask ? (postMask[gid] != 0u) : (((ball[colw] >> lane) & 1u) != 0u);
  uint32_t fIn = 0, pIn = 0, fOut = 0, pOut = 0;
  if (sel) {
    const uint4* ballV = reinterpret_cast<const uint4*>(ball);
    for (uint32_t s = inBr; s < kNslot; ++s) {
      const uint32_t g = conn[colw * kNslot + s];
      for (uint32_t j = 0; j < 2; ++j) {
        const uint4 ap = ballV[2 * g + j];
        const uint4 w = W3[((size_t)colw * kNslot + s) * kTileU4 + 32 * j + lane];
        fIn += popc4(w, ap);
        pIn += __popc(ap.x) + __popc(ap.y) + __popc(ap.z) + __popc(ap.w);
        const uint4 nap = make_uint4(~ap.x, ~ap.y, ~ap.z, ~ap.w);
        fOut += popc4(w, nap);
        pOut += __popc(nap.x) + __popc(nap.y) + __popc(nap.z) + __popc(nap.w);
      }
    }
    atomicAdd(out + 0, fIn); atomicAdd(out + 1, pIn); atomicAdd(out + 2, fOut); atomicAdd(out + 3, pOut);
    const uint32_t m = mult ? mult[gid] : 0u;
    const uint32_t b = m > 1u ? 4u : 6u;
    atomicAdd(out + b, fIn); atomicAdd(out + b + 1, pIn);
    atomicAdd(out + (m > 1u ? 8u : 9u), 1u);
  }
}

// k_indeg, src/axon.mm:566-581 and k_untouched, src/axon.mm:501-519 (which = 0 / 1)
__global__ void k_indeg_untouched(const uint4* W0, const uint4* W1, const uint4* W2, const uint4* W3, uint32_t inBr,
                                  uint32_t ncol, uint32_t which, uint32_t* out) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t colw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (colw >= ncol) return;
  uint32_t r = 0;
  for (uint32_t s = inBr; s < kNslot; ++s)
    for (uint32_t j = 0; j < 2; ++j) {
      const size_t idx = ((size_t)colw * kNslot + s) * kTileU4 + 32 * j + lane;
      const uint4 a3 = W3[idx];
      if (which == 0u) {
        r += __popc(a3.x) + __popc(a3.y) + __popc(a3.z) + __popc(a3.w);
      } else {
        const uint4 a0 = W0[idx], a1 = W1[idx], a2 = W2[idx];
        const uint32_t x[4] = {a0.x, a0.y, a0.z, a0.w}, y[4] = {a1.x, a1.y, a1.z, a1.w},
                       z[4] = {a2.x, a2.y, a2.z, a2.w}, w[4] = {a3.x, a3.y, a3.z, a3.w};
        for (int q = 0; q < 4; ++q) {
          const uint32_t v5 = ~w[q] & z[q] & ~y[q] & x[q], v6 = ~w[q] & z[q] & y[q] & ~x[q];
          r += __popc(v5 | v6);
        }
      }
    }
  out[colw * 32u + lane] = r;
}

// k_wdiag, src/axon.mm:591-638
__global__ void k_wdiag(const uint4* W0, const uint4* W1, const uint4* W2, const uint4* W3, const uint32_t* conn,
                        const uint32_t* memb, const uint32_t* asmSpk, uint32_t nstim, uint32_t inBr, uint32_t sel,
                        uint32_t ncol, uint32_t* hist) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t colw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (colw >= ncol) return;
  const uint32_t mypost = memb[colw * 32u + lane];
  if (mypost == 0u) return;
  uint32_t acc[48];
  for (int i = 0; i < 48; ++i) acc[i] = 0u;
  for (uint32_t s = 0; s < kNslot; ++s) {
    const bool isAff = s < inBr;
    if (sel == 0u && isAff) continue;
    if (sel == 1u && !isAff) continue;
    const uint32_t g = conn[colw * kNslot + s];
    for (uint32_t j = 0; j < 2; ++j) {
      const size_t idx = ((size_t)colw * kNslot + s) * kTileU4 + 32 * j + lane;
      const uint4 A0 = W0[idx], A1 = W1[idx], A2 = W2[idx], A3 = W3[idx];
      const uint32_t a0[4] = {A0.x, A0.y, A0.z, A0.w}, a1[4] = {A1.x, A1.y, A1.z, A1.w},
                     a2[4] = {A2.x, A2.y, A2.z, A2.w}, a3[4] = {A3.x, A3.y, A3.z, A3.w};
      for (int q = 0; q < 4; ++q) {
        uint32_t within = 0, anyp = 0;
        for (uint32_t qq = 0; qq < nstim; ++qq) {
          const uint32_t ap = asmSpk[(size_t)qq * ncol + 8u * g + 4u * j + q];
          anyp |= ap;
          if ((mypost >> qq) & 1u) within |= ap;
        }
        const uint32_t between = anyp & ~within;
        for (uint32_t v = 0; v < 16u; ++v) {
          const uint32_t eq = ((v & 1u) ? a0[q] : ~a0[q]) & ((v & 2u) ? a1[q] : ~a1[q]) & ((v & 4u) ? a2[q] : ~a2[q]) &
                              ((v & 8u) ? a3[q] : ~a3[q]);
          acc[v] += __popc(eq & within);
          acc[16 + v] += __popc(eq & between);
          acc[32 + v] += __popc(eq);
        }
      }
    }
  }
  for (int i = 0; i < 48; ++i)
    if (acc[i]) atomicAdd(hist + i, acc[i]);
}

// k_bstest, src/axon.mm:424-434: one thread per 32-synapse word
__global__ void k_bstest(uint32_t* A0, uint32_t* A1, uint32_t* A2, uint32_t* A3, const uint32_t* M, uint32_t op,
                         uint32_t lo, uint32_t hi, uint64_t n) {
  const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  uint32_t a0 = A0[g], a1 = A1[g], a2 = A2[g], a3 = A3[g];
  if (op == 0u) bs_inc(a0, a1, a2, a3, M[g]);
  else if (op == 1u) bs_dec(a0, a1, a2, a3, M[g]);
  else band_clip(a0, a1, a2, a3, band_of(lo, hi));  // as learn_word does
  A0[g] = a0; A1[g] = a1; A2[g] = a2; A3[g] = a3;
}

// The k-of-32 of the kernels with a lane per neuron (warp_kwta, src/axon.mm:134-144) on n columns
// of 32 values, one warp per column: out[3i..3i+2] = winners ballot, vk, vk1.
__global__ void k_kwtatest(const uint32_t* v, const uint32_t* k, uint32_t* out, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u, col = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (col >= n) return;  // whole warps
  uint32_t vk, vk1;
  const uint32_t ball = warp_kwta(v[(size_t)col * 32u + lane], lane, k[col], vk, vk1);
  if (lane == 0) {
    out[3u * col] = ball;
    out[3u * col + 1u] = vk;
    out[3u * col + 2u] = vk1;
  }
}

cudaError_t launch_wstat(const NetDev& d, uint32_t ncol, uint32_t* out, cudaStream_t st) {
  const uint64_t nU4 = (uint64_t)ncol * kNslot * kTileU4;
  k_wstat<<<148 * 8, 256, 0, st>>>(d.W3, nU4, out);
  return cudaGetLastError();
}
cudaError_t launch_within(const NetDev& d, uint32_t ncol, uint32_t inBr, uint32_t inCols, const uint32_t* ball,
                          uint32_t useMask, const uint32_t* postMask, const uint32_t* mult, uint32_t* out,
                          cudaStream_t st) {
  k_within<<<(ncol * 32 + 255) / 256, 256, 0, st>>>(d.W3, d.conn, ball, inBr, inCols, ncol, useMask, postMask, mult, out);
  return cudaGetLastError();
}
cudaError_t launch_indeg_untouched(const NetDev& d, uint32_t ncol, uint32_t inBr, uint32_t which, uint32_t* out,
                                   cudaStream_t st) {
  k_indeg_untouched<<<(ncol * 32 + 255) / 256, 256, 0, st>>>(d.W0, d.W1, d.W2, d.W3, inBr, ncol, which, out);
  return cudaGetLastError();
}
cudaError_t launch_wdiag(const NetDev& d, uint32_t ncol, const uint32_t* memb, const uint32_t* asmSpk, uint32_t nstim,
                         uint32_t inBr, uint32_t sel, uint32_t* hist, cudaStream_t st) {
  k_wdiag<<<(ncol * 32 + 127) / 128, 128, 0, st>>>(d.W0, d.W1, d.W2, d.W3, d.conn, memb, asmSpk, nstim, inBr, sel, ncol,
                                                  hist);
  return cudaGetLastError();
}
cudaError_t launch_bstest(uint32_t* a0, uint32_t* a1, uint32_t* a2, uint32_t* a3, const uint32_t* m, uint32_t op,
                          uint32_t lo, uint32_t hi, uint64_t n, cudaStream_t st) {
  k_bstest<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a0, a1, a2, a3, m, op, lo, hi, n);
  return cudaGetLastError();
}
cudaError_t launch_kwtatest(const uint32_t* v, const uint32_t* k, uint32_t* out, uint32_t n, cudaStream_t st) {
  k_kwtatest<<<(n + 7u) / 8u, 256, 0, st>>>(v, k, out, n);
  return cudaGetLastError();
}

}  // namespace axon
