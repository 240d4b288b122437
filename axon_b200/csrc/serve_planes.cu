// The recall server's step on the bit-plane readout (planes_kernel.cuh): every admitted
// trajectory of every network advances by the launch's steps, each network on a share of the
// CTAs with a barrier of its own.
#include <cstdint>

#include "plain.cuh"
#include "planes_kernel.cuh"

namespace axon {

PlanesShape planes_serve_shape(uint32_t ncol, uint32_t B, int grid, uint32_t cols, uint32_t want, PlanesCfg* c) {
  PlanesShape s{};
  s.grid = grid;
  // several teams' staged tiles don't stay in the L2 between steps (four networks of 4,096
  // columns are 680 MB), so that reading what is needed pays up to larger batches (us per step of
  // four teams, read / staged: 265 / 310 at 160 trajectories in the largest, 306 / 329 at 190, 380 / 345 at 223)
  const bool teams = cols > (ncol + (uint32_t)grid - 1u) / (uint32_t)grid;
  s.direct = B <= (teams ? 192u : kPlanesDirectB) ? 1u : 0u;
  s.smem = planes_fit(ncol, B, s.direct != 0u, true, cols, want, c);
  return s;
}

cudaError_t planes_serve_prepare(const PlanesCfg& c) {
  for (uint32_t direct = 0; direct < 2u; ++direct) {
    const cudaError_t e = raise_smem_limit(planes_fn<true>(c, direct));
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_serve_planes(const PlanesDev& d, const PlanesCfg& c, const PlanesShape& s, cudaStream_t st) {
  void* args[] = {(void*)&d, (void*)&c};
  return cudaLaunchCooperativeKernel(planes_fn<true>(c, s.direct), dim3(s.grid), dim3(planes_threads(s.direct != 0u)), args, s.smem, st);
}

}  // namespace axon
