// x passes (A, E) for complex FP32 with compile-time axis plans: the
// column-pair kernels of tile_passes.cuh instantiated for the plan of their
// axis length (tplans.inc).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include <mutex>

#include "mvp.hpp"
#include "tile_passes.cuh"

namespace bdda {
namespace tstatic {

template <class K>
cudaError_t set_smem(K kernel, int bytes, std::once_flag& once, cudaError_t& cfg) {
  std::call_once(once, [&] { cfg = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); });
  return cfg;
}

// x passes (A, E) with the plan of Px (tplans.inc)
template <class P>
cudaError_t launch_x(int pass, const TileArgs& a) {
  const MvpGeom& g = *a.g;
  const int max_nx = kMaxStaticLine / 2;
  // [2 buffers][8 columns][2 fields] lines + the occupancy of the tile
  auto smem_x2 = [](int nx) { return 4 * kTZ * P::LW * (int)sizeof(float2) + nx * kTZ * 4; };
  const int smem_ae = smem_x2(max_nx);
  int fpg = 0;
  const dim3 grid(g.ntiles, x_field_groups(a.nfield, g.ntiles, a.sms, &fpg, g.tune.xcta));
  static std::once_flag oa, oe;
  static cudaError_t ca = cudaSuccess, ce = cudaSuccess;
  cudaError_t e = cudaSuccess;
  if (pass == kTileA) {
    if ((e = set_smem(tile::k_pass_a2i<P>, smem_ae, oa, ca)) != cudaSuccess) return e;
    launch_pdl(tile::k_pass_a2i<P>, grid, kTileThreads, smem_x2(g.nx), a.st,
        a.x, a.ldx, a.nfield, fpg, g.f, g.occ, g.tiles, g.nx, g.ny, g.nz, g.nzp, g.nzt, a.twx, a.t1, a.done);
  } else {
    if ((e = set_smem(tile::k_pass_e2i<P>, smem_ae, oe, ce)) != cudaSuccess) return e;
    launch_pdl(tile::k_pass_e2i<P>, grid, kTileThreads, smem_x2(g.nx), a.st,
        a.t1, a.nfield, fpg, g.f, g.occ, g.tiles, g.nx, g.ny, g.nz, g.nzp, g.nzt, a.twx, a.x, a.ldx, a.diag, a.jpre, a.y,
        a.ldy, a.done);
  }
  return cudaGetLastError();
}

}  // namespace tstatic
}  // namespace bdda
