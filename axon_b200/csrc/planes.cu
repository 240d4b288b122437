// Host side of the bit-plane batched readout, and the kernels that prepare its layouts; the
// readout itself is in planes_kernel.cuh.
#include <cstdint>

#include "plain.cuh"
#include "planes_kernel.cuh"

namespace axon {

// One warp per tile: the eight words of its 32 rows transposed, and their row counts.
__global__ void __launch_bounds__(256) k_make_w3p(const uint4* __restrict__ W3, uint32_t* __restrict__ W3P, uint32_t ntile) {
  const uint32_t lane = threadIdx.x & 31u, tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (tile >= ntile) return;
  const uint4 a = __ldcs(W3 + (size_t)tile * kTileU4 + lane), b = __ldcs(W3 + (size_t)tile * kTileU4 + 32 + lane);
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  uint32_t* o = W3P + (size_t)tile * kPlaneTile;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t n = (uint32_t)__popc(w[i]);
    uint32_t p = 0u;
#pragma unroll
    for (uint32_t q = 0; q < 6; ++q) {
      const uint32_t v = __ballot_sync(kFull, (n >> q) & 1u);
      if (lane == q) p = v;
    }
    o[i * kPlaneBlk + lane] = transpose32(w[i], lane);
    if (lane < 8u) o[i * kPlaneBlk + 32u + lane] = p;
  }
}

// One warp per column (lane = neuron).
__global__ void k_planes_aux(const uint32_t* bias, uint32_t biasShift, const uint32_t* mult, uint32_t* biasP,
                             uint32_t* multM, uint32_t ncol) {
  const uint32_t lane = threadIdx.x & 31u, col = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (col >= ncol) return;
  if (biasP) {
    const uint32_t v = min(bias[col * 32u + lane] >> biasShift, (1u << kPlanes) - 1u);
    uint32_t p = 0u;
#pragma unroll
    for (uint32_t i = 0; i < kPlanes; ++i) {
      const uint32_t x = __ballot_sync(kFull, (v >> i) & 1u);
      if (lane == i) p = x;
    }
    if (lane < 16u) biasP[col * 16u + lane] = p;
  }
  if (multM) {
    const uint32_t x = __ballot_sync(kFull, mult[col * 32u + lane] > 1u);
    if (lane == 0) multM[col] = x;
  }
}

// The known-answer hook's second half, after k_kwtatest: where the values fit the drive planes,
// plane_kwta has to give the same winners and values; a column where it does not gets its ballot
// inverted. (With no winners, or all, the readout asks for no values.)
__global__ void k_kwtatest_planes(const uint32_t* v, const uint32_t* k, uint32_t* out, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u, col = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (col >= n) return;  // whole warps
  const uint32_t x = v[(size_t)col * 32u + lane], kk = k[col];
  if (__any_sync(kFull, x >> kPlanes)) return;
  uint32_t D[kPlanes], vk, vk1;
#pragma unroll
  for (uint32_t i = 0; i < kPlanes; ++i) D[i] = __ballot_sync(kFull, (x >> i) & 1u);
  const uint32_t ball = plane_kwta(D, kk, true, vk, vk1);
  const bool same = ball == out[3u * col] && (kk == 0u || (vk == out[3u * col + 1u] && vk1 == out[3u * col + 2u]));
  __syncwarp();
  if (lane == 0 && !same) out[3u * col] = ~ball;
}

PlanesShape planes_shape(uint32_t ncol, uint32_t B, int sms, PlanesCfg* c) {
  PlanesShape s{};
  s.grid = sms;
  // up to here the tiles that the trajectories need are read faster through L2 than whole
  // columns are staged (us per step, read / staged: 33 / 70 at 32 trajectories, 50 / 70 at 64,
  // 64 / 76 at 112, 73 / 79 at 150, 81 / 82 at 176)
  s.direct = B <= kPlanesDirectB ? 1u : 0u;
  s.smem = planes_fit(ncol, B, s.direct != 0u, false, (ncol + (uint32_t)sms - 1u) / (uint32_t)sms, (B + (uint32_t)sms - 1u) / (uint32_t)sms,
                      c);
  return s;
}

cudaError_t planes_max_blocks_per_sm(const PlanesCfg& c, const PlanesShape& s, int* out) {
  const void* fn = planes_fn<false>(c, s.direct);
  const cudaError_t e = raise_smem_limit(fn);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, fn, planes_threads(s.direct != 0u), s.smem);
}

cudaError_t launch_recall_planes(const PlanesDev& d, const PlanesCfg& c, const PlanesShape& s, cudaStream_t st) {
  void* args[] = {(void*)&d, (void*)&c};
  return cudaLaunchCooperativeKernel(planes_fn<false>(c, s.direct), dim3(s.grid), dim3(planes_threads(s.direct != 0u)), args, s.smem, st);
}

cudaError_t launch_kwtatest_planes(const uint32_t* v, const uint32_t* k, uint32_t* out, uint32_t n, cudaStream_t st) {
  k_kwtatest_planes<<<(n + 7u) / 8u, 256, 0, st>>>(v, k, out, n);
  return cudaGetLastError();
}

cudaError_t launch_make_w3p(const uint4* W3, uint32_t* W3P, uint32_t ncol, cudaStream_t st) {
  const uint32_t ntile = ncol * kNslot;
  k_make_w3p<<<(ntile + 7u) / 8u, 256, 0, st>>>(W3, W3P, ntile);
  return cudaGetLastError();
}

cudaError_t launch_planes_aux(const uint32_t* bias, uint32_t biasShift, const uint32_t* mult, uint32_t* biasP,
                              uint32_t* multM, uint32_t ncol, cudaStream_t st) {
  k_planes_aux<<<(ncol + 7u) / 8u, 256, 0, st>>>(bias, biasShift, mult, biasP, multM, ncol);
  return cudaGetLastError();
}

}  // namespace axon
