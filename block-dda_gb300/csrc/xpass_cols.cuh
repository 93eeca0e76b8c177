// x passes (A: gather and forward, E: inverse and scatter) for complex FP32
// with compile-time plans, on the column-pair stages of ypass_cols.cuh.
//
// A CTA owns an occupied (y, 8-column z tile) and walks its fields two at a
// time: eight lanes of a butterfly are the four column pairs of two fields.
// Pass A's first stage gathers the occupied sites, its last one writes T1;
// pass E's first stage reads T1, its last one scatters to the occupied sites
// (+ diag o x, o jpre).
//
// N=65536, L=32 (Px=270): A 0.915 -> 0.657 ms, E 1.15 -> 0.79 ms against line
// pairs interleaved in shared memory, one warp each (16 bytes of shared memory
// read and written per element and stage and again to fill or drain the tile);
// N=16384, L=16 (Px=160): 0.088 -> 0.068 and 0.115 -> 0.105 ms; N=8192, L=16
// (Px=128): 0.048 -> 0.034 and 0.060 -> 0.050 ms.  Bound by memory: the gather
// and scatter touch 8-byte sites, T1 streams through at its copy rate.
#pragma once

#include "ypass_cols.cuh"

namespace bdda {
namespace xcol {

constexpr int kFieldPairs = kTZ / 2;  // column pairs of one field in a tile

// Occupancy of the tile's sites -> socc[nx][kTZ] (-1: empty)
__device__ __forceinline__ void load_occ(int* socc, const int* __restrict__ occ, int y, int z0, int nx, int ny, int nz) {
  for (int i = threadIdx.x; i < nx * kTZ; i += blockDim.x) {
    const int z = z0 + (i & (kTZ - 1));
    socc[i] = z < nz ? occ[((size_t)(i / kTZ) * ny + y) * nz + z] : -1;
  }
  __syncthreads();
}

template <class P>
__global__ void __launch_bounds__(ycol::threads<P>(), ycol::min_blocks<P>())
k_pass_a(const float2* __restrict__ x, int ldx, int nfield, int fpg, int fc, const int* __restrict__ occ,
         const int* __restrict__ tiles, int nx, int ny, int nz, int nzp, int nzt, const float4* __restrict__ tw,
         float2* __restrict__ t1, const int* done) {
  pdl_begin();
  if (done && *(volatile const int*)done) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int Px = P::N, step = ycol::threads<P>() / ycol::kPairs;
  ulonglong2* tile = reinterpret_cast<ulonglong2*>(smem_raw);         // [Px][kPairs]
  int* socc = reinterpret_cast<int*>(tile + Px * ycol::kPairs);       // [nx][kTZ]
  const int t = tiles[blockIdx.x], y = t / nzt, z0 = (t - y * nzt) * kTZ;
  load_occ(socc, occ, y, z0, nx, ny, nz);
  const int c = threadIdx.x & (ycol::kPairs - 1), first = threadIdx.x / ycol::kPairs;
  const int h = c / kFieldPairs, p = c & (kFieldPairs - 1);
  const bool pval = z0 + 2 * p < nz;
  const size_t row = (size_t)ny * nzp;
  tile += c;
  const int fend = min(nfield, (int)(blockIdx.y + 1) * fpg);
  for (int f = blockIdx.y * fpg; f < fend; f += 2) {
    const int fh = f + h;
    const bool on = pval && fh < fend;
    const float2* xc = x + (size_t)(fh / fc) * ldx + fh % fc;
    float2* o = t1 + (size_t)fh * Px * row + (size_t)y * nzp + z0 + 2 * p;
    auto gather = [&](int i) {
      const int2 m = *reinterpret_cast<const int2*>(socc + i * kTZ + 2 * p);
      float2 a = make_float2(0.f, 0.f), b = a;
      if (on && m.x >= 0) a = xc[(size_t)fc * m.x];
      if (on && m.y >= 0) b = xc[(size_t)fc * m.y];
      return pk::cp{pk::p2(a.x, b.x), pk::p2(a.y, b.y)};
    };
    auto to_tile = [&](int i, pk::cp v) { pk::sts(tile + i * ycol::kPairs, v); };
    auto from_tile = [&](int i) { return pk::lds(tile + i * ycol::kPairs); };
    auto to_t1 = [&](int i, pk::cp v) {
      if (on) ycol::store_pair(o + i * row, v);
    };
    if constexpr (P::nst == 1) {
      ycol::stage<P, 0, false, step, true>(tw, first, nx, gather, to_t1);
    } else {
      ycol::stage<P, 0, false, step, true>(tw, first, nx, gather, to_tile);
      __syncthreads();
      ycol::middle<P, 1, false, step>(tile, tw, first);
      ycol::stage<P, P::nst - 1, false, step, false>(tw, first, nx, from_tile, to_t1);
      __syncthreads();
    }
  }
}

template <class P>
__global__ void __launch_bounds__(ycol::threads<P>(), ycol::min_blocks<P>())
k_pass_e(const float2* __restrict__ t1, int nfield, int fpg, int fc, const int* __restrict__ occ,
         const int* __restrict__ tiles, int nx, int ny, int nz, int nzp, int nzt, const float4* __restrict__ tw,
         const float2* __restrict__ x, int ldx, const float2* __restrict__ diag, const float2* __restrict__ jpre,
         float2* __restrict__ y, int ldy, const int* done) {
  pdl_begin();
  if (done && *(volatile const int*)done) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int Px = P::N, step = ycol::threads<P>() / ycol::kPairs;
  ulonglong2* tile = reinterpret_cast<ulonglong2*>(smem_raw);
  int* socc = reinterpret_cast<int*>(tile + Px * ycol::kPairs);
  const int t = tiles[blockIdx.x], yy = t / nzt, z0 = (t - yy * nzt) * kTZ;
  load_occ(socc, occ, yy, z0, nx, ny, nz);
  const int c = threadIdx.x & (ycol::kPairs - 1), first = threadIdx.x / ycol::kPairs;
  const int h = c / kFieldPairs, p = c & (kFieldPairs - 1);
  const bool pval = z0 + 2 * p < nz;
  const size_t row = (size_t)ny * nzp;
  tile += c;
  const int fend = min(nfield, (int)(blockIdx.y + 1) * fpg);
  for (int f = blockIdx.y * fpg; f < fend; f += 2) {
    const int fh = f + h, l = fh / fc, comp = fh - l * fc;
    const bool on = pval && fh < fend;
    const float2* g = on ? t1 + (size_t)fh * Px * row + (size_t)yy * nzp + z0 + 2 * p : t1;
    const size_t grow = on ? row : 0;  // lanes with nothing to read load one address
    auto from_t1 = [&](int i) { return ycol::load_pair(g + i * grow); };
    auto to_tile = [&](int i, pk::cp v) { pk::sts(tile + i * ycol::kPairs, v); };
    auto from_tile = [&](int i) { return pk::lds(tile + i * ycol::kPairs); };
    auto put = [&](int m, float2 v) {
      const size_t r = (size_t)fc * m + comp;
      if (diag != nullptr) v = cadd(v, cmul(diag[r], x[(size_t)l * ldx + r]));
      if (jpre != nullptr) v = cmul(v, jpre[r]);
      y[(size_t)l * ldy + r] = v;
    };
    auto scatter = [&](int i, pk::cp v) {
      const int2 m = *reinterpret_cast<const int2*>(socc + i * kTZ + 2 * p);
      float2 a, b;
      pk::unp(v.re, a.x, b.x);
      pk::unp(v.im, a.y, b.y);
      if (on && m.x >= 0) put(m.x, a);
      if (on && m.y >= 0) put(m.y, b);
    };
    if constexpr (P::nst == 1) {
      ycol::stage<P, 0, true, step, true>(tw, first, nx, from_t1, scatter);
    } else {
      ycol::stage<P, P::nst - 1, true, step, true>(tw, first, nx, from_t1, to_tile);
      __syncthreads();
      ycol::middle<P, P::nst - 2, true, step>(tile, tw, first);
      ycol::stage<P, 0, true, step, false>(tw, first, nx, from_tile, scatter);
      __syncthreads();
    }
  }
}

// x pass A or E with the plan of Px (tplans.inc: its radix sequences)
template <class P>
cudaError_t launch(int pass, const TileArgs& a) {
  const MvpGeom& g = *a.g;
  constexpr int tile = P::N * ycol::kPairs * (int)sizeof(ulonglong2);
  static std::once_flag once;
  static cudaError_t cfg = cudaSuccess;
  std::call_once(once, [] {
    const int most = tile + P::N / 2 * kTZ * (int)sizeof(int);
    for (const void* k : {(const void*)k_pass_a<P>, (const void*)k_pass_e<P>}) {
      if (cfg == cudaSuccess) cfg = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
      if (cfg == cudaSuccess) cfg = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 80);  // as the y passes
    }
  });
  if (cfg != cudaSuccess) return cfg;
  const int smem = tile + g.nx * kTZ * (int)sizeof(int);
  int fpg = 0;
  const dim3 grid(g.ntiles, x_field_groups(a.nfield, g.ntiles, a.sms, &fpg, g.tune.xcta));
  if (pass == kTileA)
    launch_pdl(k_pass_a<P>, grid, ycol::threads<P>(), smem, a.st, a.x, a.ldx, a.nfield, fpg, g.f, g.occ, g.tiles, g.nx, g.ny,
               g.nz, g.nzp, g.nzt, a.twxp, a.t1, a.done);
  else
    launch_pdl(k_pass_e<P>, grid, ycol::threads<P>(), smem, a.st, a.t1, a.nfield, fpg, g.f, g.occ, g.tiles, g.nx, g.ny, g.nz,
               g.nzp, g.nzt, a.twxp, a.x, a.ldx, a.diag, a.jpre, a.y, a.ldy, a.done);
  return cudaGetLastError();
}

}  // namespace xcol
}  // namespace bdda
