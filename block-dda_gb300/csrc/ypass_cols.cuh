// y passes (B: forward, D: inverse) for complex FP32 with compile-time plans.
//
// A task is 16 z-columns of one (field, x) plane: a thread owns one pair of
// adjacent columns and walks butterflies along y in the two lanes of f32x2
// instructions (pfft.cuh).  The first stage reads its elements from global
// memory and the last one writes them back -- a row of 16 columns is one
// 128-byte segment either way -- so a line passes through shared memory once
// per stage boundary: 16 bytes per element and boundary, where filling and
// draining a tile around in-place stages took 64 to 80.  Shared memory holds
// the tile as rows of eight 16-byte pairs, so that eight lanes always cover a
// 128-byte row whatever the stage's stride is (no bank conflicts, no padding),
// and the eight lanes of a butterfly share its twiddles.
//
// N=65536, L=32 (Py=270, three stages; 7.9 GB, 1.17 ms at the measured copy
// rate): forward 2.40 -> 2.09 ms, inverse 2.72 -> 1.62 ms; N=16384, L=16
// (Py=160, two stages): 0.224 -> 0.174 and 0.240 -> 0.171 ms.  Both wait for
// memory: the forward pass gains from a prefetched next task (2.63 -> 2.09; its
// first stage has few rows to read per thread), the inverse does not (1.62 ->
// 1.81; the second buffer costs a resident CTA), so the autotuner picks it for
// each, and the defaults are what these sizes took.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "mvp.hpp"
#include "pdl.cuh"
#include "pfft.cuh"
#include "static_fft.cuh"
#include "tile_passes.cuh"

namespace bdda {
namespace ycol {

constexpr int kCols = 16;           // z-columns per task
constexpr int kPairs = kCols / 2;   // threads of one butterfly
constexpr int kLoads = 8;           // elements a thread reads from global memory before it transforms them

template <class P>
constexpr int max_radix() {
  int m = 0;
  for (int s = 0; s < P::nst; ++s) m = P::rad[s] > m ? P::rad[s] : m;
  return m;
}
// Threads per SM to compile for: 1024 (64 registers), 768 for radices above 10, whose pair butterflies take four
// registers an element.  N=65536, L=32 at 768 / 512 threads instead: forward 2.11 -> 2.09, inverse 1.75 -> 1.62 ms;
// Py=160 (10 x 16): forward 0.180 -> 0.174 ms.
template <class P>
constexpr int sm_threads() { return max_radix<P>() > 10 ? 768 : 1024; }
// Shared memory of an SM, and what a CTA takes beside its tile.
constexpr int kSmemSm = 228 * 1024, kSmemCta = 1024;
// Threads per CTA: the multiple of 32 with the least idling over a stage's 8 N / R butterfly threads, weighted by the
// stages' work, over the threads, up to 896, that the tiles fitting an SM make.  Without the second factor 288 = 9 2 16
// took 64 threads, three CTAs of them for each six tiles' room (y 7.9, x 9.7 ps per point for both directions; with it 5.9
// and 7.1), 360 = 2 12 15 likewise (9.0 / 13.9 -> 7.1 / 7.1).
template <class P>
constexpr int threads() {
  int best = 64;
  long cost = -1;
  for (int t = 64; t <= 384; t += 32) {
    long c = 0;
    for (int s = 0; s < P::nst; ++s) {
      const int items = kPairs * (P::N / P::rad[s]);
      c += (long)((items + t - 1) / t) * t * P::rad[s];
    }
    const int room = kSmemSm / (P::N * kCols * 8 + kSmemCta), ctas = std::min(sm_threads<P>() / t, room);
    c = c * 896 / std::min(ctas * t, 896);
    if (cost < 0 || c <= cost) { best = t; cost = c; }
  }
  return best;
}
template <class P>
constexpr int min_blocks() { return sm_threads<P>() / threads<P>(); }

// Rows a task reads, at most.
template <class P, bool INV>
__host__ __device__ constexpr int in_rows() { return INV ? P::N : (P::N + 1) / 2; }

__device__ __forceinline__ pk::cp load_pair(const float2* p) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(p));
  return {pk::p2(v.x, v.z), pk::p2(v.y, v.w)};
}
__device__ __forceinline__ void store_pair(float2* p, pk::cp v) {
  float4 o;
  pk::unp(v.re, o.x, o.z);
  pk::unp(v.im, o.y, o.w);
  *reinterpret_cast<float4*>(p) = o;
}

// One stage of a column pair: butterflies u = first + k STEP of stage s, element idx read by load(idx) and written by
// store(idx, value).  Forward first stage / inverse last stage: only idx < nv are read / written (nv <= N / 2, so
// elements 2 i >= R never are).  U butterflies are loaded before the first is transformed.
template <class P, int s, bool INV, int STEP, bool GLOBAL, class Load, class Store>
__device__ __forceinline__ void stage(const float4* __restrict__ tw, int first, int nv, Load load, Store store) {
  constexpr int R = P::rad[s], M = P::M(s), Ls = M * R, B = P::N / R;
  constexpr bool prune_in = !INV && s == 0;
  constexpr int RL = prune_in ? (R + 1) / 2 : R;  // elements read
  constexpr int rounds = (B + STEP - 1) / STEP;
  constexpr int U = GLOBAL ? (kLoads / RL < 1 ? 1 : kLoads / RL < rounds ? kLoads / RL : rounds) : 1;
  for (int u0 = first; u0 < B; u0 += U * STEP) {
    pk::cp w[U][RL];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int u = u0 + j * STEP, b = u / M, n1 = u - b * M, idx0 = b * Ls + n1;
#pragma unroll
      for (int i = 0; i < RL; ++i)
        if (u < B && (!prune_in || idx0 + i * M < nv)) w[j][i] = load(idx0 + i * M);
        else w[j][i] = pk::cp{0ull, 0ull};
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int u = u0 + j * STEP;
      if (u >= B) break;
      const int b = u / M, n1 = u - b * M, idx0 = b * Ls + n1;
      pk::cp v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = i < RL ? w[j][i] : pk::cp{0ull, 0ull};
      const float4* tws = tw + P::TWO(s) + n1;
      if constexpr (INV && M > 1) {
#pragma unroll
        for (int k = 1; k < R; ++k) {
          pk::u64 c, sn;
          pk::ld_tw(tws + (k - 1) * M, c, sn);
          v[k] = pk::tw_mulc(v[k], c, sn);
        }
      }
      pk::dft<R, INV>(v);
      if constexpr (!INV && M > 1) {
#pragma unroll
        for (int k = 1; k < R; ++k) {
          pk::u64 c, sn;
          pk::ld_tw(tws + (k - 1) * M, c, sn);
          v[k] = pk::tw_mul(v[k], c, sn);
        }
      }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (INV && s == 0 && (2 * i >= R || idx0 + i * M >= nv)) continue;
        store(idx0 + i * M, v[i]);
      }
    }
  }
}

// Stages between the first and the last, in shared memory, a barrier after each.
template <class P, int s, bool INV, int STEP>
__device__ __forceinline__ void middle(ulonglong2* tile, const float4* tw, int first) {
  if constexpr (s > 0 && s < P::nst - 1) {
    stage<P, s, INV, STEP, false>(tw, first, 0, [&](int i) { return pk::lds(tile + i * kPairs); },
                     [&](int i, pk::cp v) { pk::sts(tile + i * kPairs, v); });
    __syncthreads();
    middle<P, INV ? s - 1 : s + 1, INV, STEP>(tile, tw, first);
  }
}

// B: T1[f][x][y < ny][z] -> T2[f][x][Py][z] (rows of empty tiles read as zero)
// D: T2[f][x][Py][z] -> T1[f][x][y < ny][z] (rows of listed tiles written)
// NBUF = 2: the rows of a CTA's next task are copied to a second shared buffer by cp.async while it works on the
// current one's later stages.
template <bool INV, class P, int NBUF>
__global__ void __launch_bounds__(threads<P>(), min_blocks<P>())
k_pass_y(const float2* __restrict__ src, float2* __restrict__ dst, const unsigned char* __restrict__ tmask, int ny, int nz,
         int nzp, int nzt, int ntask, const float4* __restrict__ tw, const int* done) {
  // many uneven tasks per CTA: the z pass takes the SMs as they run out of them (24 x 24 x 225 box, L=16, 459 -> 443 us)
  if (ntask >= 4 * (int)gridDim.x) pdl_trigger();
  pdl_begin();
  if (done && *(volatile const int*)done) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int Py = P::N, T = threads<P>(), step = T / kPairs;
  constexpr int s0 = INV ? P::nst - 1 : 0, s1 = INV ? 0 : P::nst - 1;
  ulonglong2* tile = reinterpret_cast<ulonglong2*>(smem_raw);       // [Py][kPairs]
  float4* next = reinterpret_cast<float4*>(tile + Py * kPairs);     // [rows read][kPairs], NBUF = 2
  unsigned* mask = reinterpret_cast<unsigned*>(next + (NBUF == 2 ? in_rows<P, INV>() * kPairs : 0));  // [ny][mw] listed tiles
  const int c = threadIdx.x & (kPairs - 1), first = threadIdx.x / kPairs;
  const int nin = INV ? Py : ny, nout = INV ? ny : Py;
  const int mw = (nzt + 31) / 32, nzt2 = (nz + kCols - 1) / kCols;
  for (int k = threadIdx.x; k < ny * mw; k += T) {
    const int y = k / mw, t0 = (k - y * mw) * 32;
    unsigned m = 0;
    for (int t = t0; t < min(nzt, t0 + 32); ++t) m |= (tmask[(size_t)y * nzt + t] ? 1u : 0u) << (t - t0);
    mask[k] = m;
  }
  __syncthreads();
  tile += c;
  next += c;
  struct Task { int r, z; bool zval; };
  // adjacent z tiles in adjacent CTAs: the 128-byte pieces of a T1 / T2 row move at the same time
  auto task_of = [&](int t) {
    const int r = t / nzt2, z = (t - r * nzt2) * kCols + 2 * c;  // r = f * Px + x
    return Task{r, z, z < nz};
  };
  auto listed = [&](int i, int z) { return ((mask[i * mw + z / (32 * kTZ)] >> (z / kTZ & 31)) & 1u) != 0; };
  auto issue = [&](const Task& k) {
    const float2* g = src + (size_t)k.r * nin * nzp + k.z;
    for (int i = first; i < nin; i += step) {
      const bool ok = k.zval && (INV || listed(i, k.z));
      bdda::tile::cp_async<16>(next + i * kPairs, ok ? g + i * nzp : src, ok);
    }
    bdda::tile::cp_commit();
  };
  if (NBUF == 2 && blockIdx.x < ntask) issue(task_of(blockIdx.x));
  for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
    const Task k = task_of(t);
    const float2* g = src + (size_t)k.r * nin * nzp + k.z;
    float2* o = dst + (size_t)k.r * nout * nzp + k.z;
    auto from_global = [&](int i) {
      const bool ok = k.zval && (INV || listed(i, k.z));
      const pk::cp v = load_pair(ok ? g + i * nzp : src);  // a load either way: a branch would keep the loads apart
      return pk::cp{ok ? v.re : 0ull, ok ? v.im : 0ull};
    };
    auto from_next = [&](int i) {
      const float4 v = next[i * kPairs];
      return pk::cp{pk::p2(v.x, v.z), pk::p2(v.y, v.w)};
    };
    auto to_tile = [&](int i, pk::cp v) { pk::sts(tile + i * kPairs, v); };
    auto from_tile = [&](int i) { return pk::lds(tile + i * kPairs); };
    auto to_global = [&](int i, pk::cp v) {
      if (k.zval && (!INV || listed(i, k.z))) store_pair(o + i * nzp, v);
    };
    if constexpr (P::nst == 1) {
      stage<P, 0, INV, step, true>(tw, first, ny, from_global, to_global);
    } else {
      if constexpr (NBUF == 2) {
        bdda::tile::cp_wait<0>();
        __syncthreads();
        stage<P, s0, INV, step, false>(tw, first, ny, from_next, to_tile);
      } else {
        stage<P, s0, INV, step, true>(tw, first, ny, from_global, to_tile);
      }
      __syncthreads();
      if (NBUF == 2 && t + gridDim.x < ntask) issue(task_of(t + gridDim.x));
      middle<P, INV ? s0 - 1 : 1, INV, step>(tile, tw, first);
      stage<P, s1, INV, step, false>(tw, first, ny, from_tile, to_global);
      if (NBUF == 1) __syncthreads();
    }
  }
}

template <class P, bool INV, int NBUF>
cudaError_t launch_buf(const TileArgs& a, int waves, int ntask) {
  const MvpGeom& g = *a.g;
  // the tile, the next task's rows, and the mask: ny <= N / 2 rows of nzt <= kMaxLine / 2 / kTZ tiles
  constexpr int smem = (P::N + (NBUF == 2 ? in_rows<P, INV>() : 0)) * kPairs * (int)sizeof(ulonglong2) +
                       P::N / 2 * ((kMaxLine / 2 / kTZ + 31) / 32) * 4;
  static std::once_flag once;
  static cudaError_t cfg = cudaSuccess;
  static int resident = 1;  // CTAs that fit on one SM
  std::call_once(once, [] {
    cfg = cudaFuncSetAttribute(k_pass_y<INV, P, NBUF>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    // 80% of the SM for shared memory, near what the other passes run with: an SM has to drain before its split changes,
    // which costs concurrent solves (three streams of N=16384, L=16 MVPs: 1.24 -> 1.11 ms each; one stream 1.157 -> 1.167)
    if (cfg == cudaSuccess) cfg = cudaFuncSetAttribute(k_pass_y<INV, P, NBUF>, cudaFuncAttributePreferredSharedMemoryCarveout, 80);
    int nb = 0;
    if (cfg == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pass_y<INV, P, NBUF>, threads<P>(), smem) == cudaSuccess && nb > 0)
      resident = nb;
  });
  if (cfg != cudaSuccess) return cfg;
  launch_pdl(k_pass_y<INV, P, NBUF>, std::min(ntask, waves * resident * a.sms), threads<P>(), smem, a.st,
      INV ? a.t2 : a.t1, INV ? a.t1 : a.t2, g.tmask, g.ny, g.nz, g.nzp, g.nzt, ntask, a.twyp, a.done);
  return cudaGetLastError();
}

template <class P, bool INV>
cudaError_t launch_dir(const TileArgs& a) {
  const MvpGeom& g = *a.g;
  const int nbuf = INV && g.tune.ybufd > 0 ? g.tune.ybufd : g.tune.ybuf;
  const int waves = INV && g.tune.ywavesd > 0 ? g.tune.ywavesd : g.tune.ywaves;
  const int ntask = a.nfield * g.Px * ((g.nz + kCols - 1) / kCols);
  // one tile where a CTA has a single task: nothing to overlap, and more CTAs fit
  if (nbuf == 1 || ntask <= 2 * a.sms) return launch_buf<P, INV, 1>(a, waves, ntask);
  return launch_buf<P, INV, 2>(a, waves, ntask);
}

// y pass B or D with the plan of Py (yplans.inc: its radix sequences)
template <class P>
cudaError_t launch(int pass, const TileArgs& a) {
  return pass == kTileB ? launch_dir<P, false>(a) : launch_dir<P, true>(a);
}

}  // namespace ycol
}  // namespace bdda
