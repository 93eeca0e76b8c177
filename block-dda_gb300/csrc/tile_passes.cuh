// Strided passes of the block MVP (A: x-forward gather, B: y-forward,
// D: y-inverse, E: x-inverse scatter).
//
// k_pass_a / k_pass_y / k_pass_e: runtime axis plans (fft_core.cuh, skewed
// layout of the plan; every precision).  A CTA stages 8 z-columns (one line
// per warp) of one tile in shared memory; forward transforms read only the
// first nv inputs.
// (Complex FP32 lines with a compile-time plan: xpass_cols.cuh, ypass_cols.cuh.)
#pragma once

#include <cuda_runtime.h>

#include "fft_core.cuh"
#include "mvp.hpp"
#include "pdl.cuh"
#include "static_fft.cuh"

namespace bdda {
namespace tile {

template <typename C>
struct RtLine {
  AxisPlan p;
  __device__ __forceinline__ int n() const { return p.N; }
  __device__ __forceinline__ int lw() const { return plan_lw<C>(p); }
  __device__ __forceinline__ int addr(int i) const { return skw(i, plan_sk<C>(p)); }
  template <bool INV>
  __device__ __forceinline__ void fft(C* line, const C* tw, int lane, int nv) const {
    if (!INV) warp_fft_lines<false, 1>(line, 0, tw, p, lane, 32, nv);
    else warp_fft_lines<true, 1>(line, 0, tw, p, lane);
  }
};


// ---- cp.async helpers (LDGSTS: global -> shared without registers) --------
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int sz = valid ? BYTES : 0;  // src-size 0: nothing read, destination zero-filled
  static_assert(BYTES == 4 || BYTES == 8 || BYTES == 16, "cp.async sizes");
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(sz) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(gmem), "n"(BYTES), "r"(sz) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ bool skip(const int* done) { return done && *(volatile const int*)done; }

// Rows of a tile one thread visits: rows r, r + kRowStep, ... in column tid % kTZ.
constexpr int kRowStep = kTileThreads / kTZ;

// ---------------------------------------------------------------- pass A
// One CTA per listed (y, z-tile): warp w owns z = z0 + w; loops over fields.
template <typename T, class Line>
__global__ void __launch_bounds__(kTileThreads)
k_pass_a(const typename cplx<T>::type* __restrict__ x, int ldx, int nfield, int fpg, int fc, const int* __restrict__ occ,
         const int* __restrict__ tiles, int nx, int ny, int nz, int nzp, int nzt, Line lay,
         const typename cplx<T>::type* __restrict__ twx, typename cplx<T>::type* __restrict__ t1, int nbuf,
         const int* done) {
  using C = typename cplx<T>::type;
  if (skip(done)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Px = lay.n();
  const int lw = lay.lw();
  C* lines = reinterpret_cast<C*>(smem_raw);                       // [nbuf][kTZ][lw]
  int* socc = reinterpret_cast<int*>(lines + nbuf * kTZ * lw);     // [nx][kTZ]
  const int tile = tiles[blockIdx.x];
  const int y = tile / nzt, z0 = (tile - y * nzt) * kTZ;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tw8 = tid & (kTZ - 1), tq = tid / kTZ;  // tile column and first row of this thread
  const bool zval = z0 + tw8 < nz;
  for (int idx = tid; idx < nx * kTZ; idx += kTileThreads) {
    const int xi = idx >> 3, w = idx & 7, z = z0 + w;
    socc[idx] = z < nz ? occ[((size_t)xi * ny + y) * nz + z] : -1;
  }
  __syncthreads();
  const size_t rowstride = (size_t)ny * nzp;  // T1 stride between x rows
  const int f0 = blockIdx.y * fpg, fend = min(nfield, f0 + fpg);  // this CTA's fields (f0 even)
  int l = f0 / fc, c = f0 - (f0 / fc) * fc;
  for (int f = f0; f < fend; ++f) {
    const int buf = nbuf == 2 ? (f & 1) : 0;
    C* line = lines + (buf * kTZ + warp) * lw;
    const C* xc = x + (size_t)l * ldx + c;
    for (int xi = lane; xi < nx; xi += 32) {
      const int m = socc[xi * kTZ + warp];
      line[lay.addr(xi)] = m >= 0 ? xc[fc * (size_t)m] : czero<C>();
    }
    __syncwarp();
    lay.template fft<false>(line, twx, lane, nx);
    __syncthreads();
    // drain: thread tid writes column w = tid % 8 of rows q = tid / 8 + 32 k
    if (zval) {
      const C* lb = lines + (buf * kTZ + tw8) * lw;
      C* out = t1 + (size_t)f * Px * rowstride + (size_t)y * nzp + z0 + tw8 + (size_t)tq * rowstride;
      for (int q = tq; q < Px; q += kRowStep, out += kRowStep * rowstride) *out = lb[lay.addr(q)];
    }
    if (nbuf == 1) __syncthreads();  // the next field's gather overwrites the drained buffer
    if (++c == fc) { c = 0; ++l; }
  }
}

// ---------------------------------------------------------------- pass B / D
// Persistent CTAs over tasks (field, x, z-tile); lines along y.
// B: T1[f][q][y<ny][z] -> T2[f][q][Py][z]   (rows of empty tiles zero-filled)
// D: T2[f][q][Py][z]   -> T1[f][q][y<ny][z] (rows of listed tiles only)
template <typename T, bool INV, class Line>
__global__ void __launch_bounds__(kTileThreads)
k_pass_y(const typename cplx<T>::type* __restrict__ src, typename cplx<T>::type* __restrict__ dst,
         const unsigned char* __restrict__ tmask, int ny, int nz, int nzp, int nzt, int ntask, Line lay,
         const typename cplx<T>::type* __restrict__ twy, int nbuf, const int* done) {
  using C = typename cplx<T>::type;
  if (skip(done)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Py = lay.n();
  const int lw = lay.lw();
  C* lines = reinterpret_cast<C*>(smem_raw);  // [nbuf][kTZ][lw]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nin = INV ? Py : ny;    // rows read
  const int nout = INV ? ny : Py;   // rows written
  const size_t in_rows = (size_t)nin, out_rows = (size_t)nout;

  const int tw8 = tid & (kTZ - 1), ty = tid / kTZ;  // tile column and first row of this thread
  // fill: thread tid loads column w = tid % 8 of rows yy = tid / 8 + 32 k (zero-filled outside the data)
  auto issue = [&](int task, int buf) {
    const int zt = task % nzt;
    const int r = task / nzt;  // f * Px + q
    const int z0 = zt * kTZ;
    const bool zval = z0 + tw8 < nz;
    const C* g = src + (size_t)r * in_rows * nzp + z0 + tw8 + (size_t)ty * nzp;
    const unsigned char* tm = tmask + zt + (size_t)ty * nzt;
    C* lb = lines + (buf * kTZ + tw8) * lw;
    for (int yy = ty; yy < nin; yy += kRowStep, g += (size_t)kRowStep * nzp, tm += (size_t)kRowStep * nzt) {
      const bool valid = zval && (INV || *tm);
      cp_async<sizeof(C)>(lb + lay.addr(yy), valid ? g : src, valid);
    }
    cp_commit();
  };

  int task = blockIdx.x;
  if (nbuf == 2 && task < ntask) issue(task, 0);
  for (int it = 0; task < ntask; ++it, task += gridDim.x) {
    const int buf = nbuf == 2 ? (it & 1) : 0;
    const int next = task + gridDim.x;
    if (nbuf == 1) {
      issue(task, 0);
      cp_wait<0>();
    } else if (next < ntask) {
      issue(next, buf ^ 1);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    __syncthreads();
    C* line = lines + (buf * kTZ + warp) * lw;
    lay.template fft<INV>(line, twy, lane, ny);
    __syncthreads();
    const int zt = task % nzt;
    const int r = task / nzt;
    const int z0 = zt * kTZ;
    if (z0 + tw8 < nz) {
      C* ob = dst + (size_t)r * out_rows * nzp + z0 + tw8 + (size_t)ty * nzp;
      const unsigned char* tm = tmask + zt + (size_t)ty * nzt;
      const C* lb = lines + (buf * kTZ + tw8) * lw;
      for (int yy = ty; yy < nout; yy += kRowStep, ob += (size_t)kRowStep * nzp, tm += (size_t)kRowStep * nzt)
        if (!INV || *tm) *ob = lb[lay.addr(yy)];
    }
    __syncthreads();  // buffer 'buf' is the cp.async target of the next-but-one task
  }
}

// ---------------------------------------------------------------- pass E
// One CTA per listed (y, z-tile); loops over fields with the next field's
// tile prefetched by cp.async; scatters the occupied sites.
template <typename T, class Line>
__global__ void __launch_bounds__(kTileThreads)
k_pass_e(const typename cplx<T>::type* __restrict__ t1, int nfield, int fpg, int fc, const int* __restrict__ occ,
         const int* __restrict__ tiles, int nx, int ny, int nz, int nzp, int nzt, Line lay,
         const typename cplx<T>::type* __restrict__ twx, const typename cplx<T>::type* __restrict__ x, int ldx,
         const typename cplx<T>::type* __restrict__ diag, const typename cplx<T>::type* __restrict__ jpre,
         typename cplx<T>::type* __restrict__ y, int ldy, int nbuf, const int* done) {
  using C = typename cplx<T>::type;
  if (skip(done)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Px = lay.n();
  const int lw = lay.lw();
  C* lines = reinterpret_cast<C*>(smem_raw);                       // [nbuf][kTZ][lw]
  int* socc = reinterpret_cast<int*>(lines + nbuf * kTZ * lw);     // [nx][kTZ]
  const int tile = tiles[blockIdx.x];
  const int yy = tile / nzt, z0 = (tile - yy * nzt) * kTZ;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t rowstride = (size_t)ny * nzp;
  for (int idx = tid; idx < nx * kTZ; idx += kTileThreads) {
    const int xi = idx >> 3, w = idx & 7, z = z0 + w;
    socc[idx] = z < nz ? occ[((size_t)xi * ny + yy) * nz + z] : -1;
  }
  const int tw8 = tid & (kTZ - 1), tq = tid / kTZ;  // tile column and first row of this thread
  const bool zval = z0 + tw8 < nz;
  // fill: thread tid loads column w = tid % 8 of rows q = tid / 8 + 32 k (zero-filled past nz)
  auto issue = [&](int f, int buf) {
    const C* g = t1 + (size_t)f * Px * rowstride + (size_t)yy * nzp + z0 + tw8 + (size_t)tq * rowstride;
    C* lb = lines + (buf * kTZ + tw8) * lw;
    for (int q = tq; q < Px; q += kRowStep, g += (size_t)kRowStep * rowstride)
      cp_async<sizeof(C)>(lb + lay.addr(q), zval ? g : t1, zval);
    cp_commit();
  };
  const int f0 = blockIdx.y * fpg, fend = min(nfield, f0 + fpg);  // this CTA's fields (f0 even)
  if (nbuf == 2) issue(f0, 0);
  int l = f0 / fc, c = f0 - (f0 / fc) * fc;
  for (int f = f0; f < fend; ++f) {
    const int buf = nbuf == 2 ? (f & 1) : 0;
    if (nbuf == 1) {
      issue(f, 0);
      cp_wait<0>();
    } else if (f + 1 < fend) {
      issue(f + 1, buf ^ 1);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    __syncthreads();
    C* line = lines + (buf * kTZ + warp) * lw;
    lay.template fft<true>(line, twx, lane, nx);
    for (int xi = lane; xi < nx; xi += 32) {
      const int m = socc[xi * kTZ + warp];
      if (m < 0) continue;
      const size_t r = fc * (size_t)m + c;
      C v = line[lay.addr(xi)];
      if (diag != nullptr) v = cadd(v, cmul(diag[r], x[(size_t)l * ldx + r]));
      if (jpre != nullptr) v = cmul(v, jpre[r]);
      y[(size_t)l * ldy + r] = v;
    }
    __syncthreads();  // buffer 'buf' is the cp.async target of field f + 2
    if (++c == fc) { c = 0; ++l; }
  }
}

// Dynamic shared memory of a runtime-plan strided pass with nbuf tile buffers
// (nx > 0: the x passes' occupancy table of the tile).
template <typename T> int smem_tile(int lw, int nx, int nbuf = 2) {
  return nbuf * kTZ * lw * (int)sizeof(typename cplx<T>::type) + nx * kTZ * 4;
}
// Two tile buffers where they fit in a CTA's shared memory, else one.
template <typename T> int tile_buffers(int lw, int nx) { return smem_tile<T>(lw, nx, 2) <= kZSmemMax ? 2 : 1; }

}  // namespace tile
}  // namespace bdda
