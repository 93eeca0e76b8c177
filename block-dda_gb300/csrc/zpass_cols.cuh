// Fused z pass (pass C) for complex FP32, f = 3, lines shorter than
// kFusedWideMinN (two or three stages of radices <= 16).
//
// A CTA takes NT tasks ((x, y) line, right-hand side or pair of them), three
// component lines each, and spreads every step's butterflies over all its
// threads: the first stage reads T2 and writes shared memory; the middle step
// (last forward stage, Green product, first inverse stage: one butterfly of
// the three components per thread, as sfft::middle3) reads and writes it once;
// the last inverse stage writes T2.  One warp per task left the middle step
// with N / R_last butterflies for 32 lanes (8 at 128 = 8 16, 10 at 150 = 10
// 15, 12 at 180 = 12 15), so those lengths ran it as three separate sweeps.
//
// PAIR: a task is two right-hand sides, transformed by the outer stages in the
// two lanes of f32x2 instructions (pfft.cuh) with shared twiddles and
// 16-byte shared-memory elements {a, b}; the middle step takes 6 R_last
// registers of line values per right-hand side and stays unpacked.  An odd last
// right-hand side runs alone in its pair.
//
// Shared memory: element q R_last + r of a line at q S + r with S odd, lines
// LW apart, LW = R_last (mod 16): the outer stages' lanes (adjacent r) and the
// middle step's (adjacent q) hit distinct banks.
//
// Bound by issue and latency (T2 at its copy rate would take 2.4 ps per point).
// Lines of 9216 (x, y) and L = 16 right-hand sides, ms, one warp per pair of
// right-hand sides -> now: 64
// 0.127 -> 0.085, 80 0.154 -> 0.121, 90 0.154 -> 0.139, 96 0.183 -> 0.132, 100
// 0.194 -> 0.158, 120 0.195 -> 0.171, 128 0.220 -> 0.168, 135 0.287 -> 0.192,
// 144 0.268 -> 0.190, 150 0.251 -> 0.205, 160 0.261 -> 0.205, 180 0.388 -> 0.278.
// The L1 data pipe is 86% busy (120 = 15 8): twiddles are loaded as 8 bytes and
// duplicated in registers (as 16-byte pairs 150 took 0.215, 180 0.290).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "mvp.hpp"
#include "pdl.cuh"
#include "pfft.cuh"
#include "static_fft.cuh"

namespace bdda {
namespace zcol {

template <class P> constexpr bool supported() { return P::N < kFusedWideMinN && fused_z(P::N, P::nst, P::Rl); }

// The plan of these kernels: the operator's, but two-stage lines take the
// radices that z_col_last_radix (mvp.hpp) gives.  The last-radix-major spectrum of a
// two-stage line is in natural order (frequency b + R0 i at i R0 + b), so it
// does not depend on which two radices the kernel uses.
template <class P, bool TWO = P::nst == 2> struct Own { using type = P; };
template <class P> struct Own<P, true> {
  static constexpr int Rl = z_col_last_radix(P::N);
  using type = sfft::Plan<P::N, 0, 0, P::N / Rl, Rl>;
};

// Line layout
template <class P> struct Lay {
  static constexpr int S = P::Rl | 1, B = P::N / P::Rl;
  static constexpr int LW = B * S + (((P::Rl - B * S) % 16) + 16) % 16;
  __device__ static __forceinline__ int addr(int idx) { return (idx / P::Rl) * S + idx % P::Rl; }
  // distance of a butterfly's elements in stage s before the last
  static constexpr int off(int s) { return (P::M(s) / P::Rl) * S; }
};

// ---- tasks and threads of a CTA -------------------------------------------------
constexpr int kSmemSm = 228 * 1024, kSmemCta = 1024;  // shared memory of an SM, and what a CTA takes beside its lines
constexpr int kMaxTasks = 4;  // 32-point lines 0.098 / 0.080 / 0.050 ms at 1 / 2 / 4; long lines take one or two
struct Task {
  long long src;   // first line in T2
  long long rhs;   // from one right-hand side of a pair to the other
  long long gl;    // Green line
  int n;           // right-hand sides (0: none)
};
template <class P, bool PAIR> constexpr int elem() { return PAIR ? 16 : 8; }
template <class P, bool PAIR> constexpr int smem_bytes(int nt) {
  return nt * (3 * Lay<P>::LW * elem<P, PAIR>() + (int)sizeof(Task));
}
// Threads per SM to compile for: a thread's line values decide its registers (144 = 16 9, ms at 768 / 512 / 384 threads:
// 0.30 / 0.201 / 0.217; 128 = 8 16: - / 0.211 / 0.190).
template <class P, bool PAIR> constexpr int sm_threads() {
  int r = 6 * P::Rl;
  for (int s = 0; s + 1 < P::nst; ++s) r = std::max(r, (PAIR ? 4 : 2) * P::rad[s]);
  return r > 64 ? 384 : r > 36 ? 512 : 768;
}
// Idle-weighted work of nt tasks on t threads, per task and resident thread.
template <class P, bool PAIR> constexpr long cost(int nt, int t) {
  const int rhs = PAIR ? 2 : 1;
  long c = 0;
  for (int s = 0; s + 1 < P::nst; ++s) {
    const int items = nt * 3 * (P::N / P::rad[s]);
    c += (long)((items + t - 1) / t) * t * P::rad[s] * 32 * rhs;
  }
  const int items = nt * rhs * (P::N / P::Rl);
  c += (long)((items + t - 1) / t) * t * P::Rl * 100;
  const int ctas = std::min(sm_threads<P, PAIR>() / t, kSmemSm / (smem_bytes<P, PAIR>(nt) + kSmemCta));
  if (ctas < 1) return 1l << 60;
  return c * 64 / nt / std::min(ctas * t, 768);
}
// Threads for nt tasks; tasks of a full CTA.
template <class P, bool PAIR> constexpr int threads(int nt) {
  int best = 32;
  for (int t = 32; t <= 256; t += 32)
    if (cost<P, PAIR>(nt, t) <= cost<P, PAIR>(nt, best)) best = t;
  return best;
}
template <class P, bool PAIR> constexpr int tasks() {
  int best = 1;
  for (int nt = 2; nt <= kMaxTasks; ++nt)
    if (cost<P, PAIR>(nt, threads<P, PAIR>(nt)) < cost<P, PAIR>(best, threads<P, PAIR>(best))) best = nt;
  return best;
}

// ---- line elements: one right-hand side, or a pair ----------------------------
template <bool PAIR> struct El;
template <> struct El<false> {
  using V = float2;   // in registers
  using E = float2;   // in shared memory
  static __device__ __forceinline__ V zero() { return make_float2(0.f, 0.f); }
  static __device__ __forceinline__ V get(const E* p) { return *p; }
  static __device__ __forceinline__ void put(E* p, V v) { *p = v; }
  static __device__ __forceinline__ V load(const float2* g, long long) { return *g; }
  static __device__ __forceinline__ void store(float2* g, long long, int, V v) { *g = v; }
  template <int R, bool INV> static __device__ __forceinline__ void fft(V* v) { dft<R, INV>(v); }
  template <bool CONJ> static __device__ __forceinline__ V tw(V v, const float2* p) {
    const float2 w = ldg_c(p);
    return CONJ ? cmulc(v, w) : cmul(v, w);
  }
};
template <> struct El<true> {
  using V = pk::cp;
  using E = float4;  // {a.re, a.im, b.re, b.im}
  static __device__ __forceinline__ V zero() { return V{0ull, 0ull}; }
  static __device__ __forceinline__ V get(const E* p) {
    const float4 v = *p;
    return V{pk::p2(v.x, v.z), pk::p2(v.y, v.w)};
  }
  static __device__ __forceinline__ void put(E* p, V v) {
    float4 o;
    pk::unp(v.re, o.x, o.z);
    pk::unp(v.im, o.y, o.w);
    *p = o;
  }
  static __device__ __forceinline__ V load(const float2* g, long long rhs) {
    const float2 a = *g, b = g[rhs];
    return V{pk::p2(a.x, b.x), pk::p2(a.y, b.y)};
  }
  static __device__ __forceinline__ void store(float2* g, long long rhs, int n, V v) {
    float2 a, b;
    pk::unp(v.re, a.x, b.x);
    pk::unp(v.im, a.y, b.y);
    *g = a;
    if (n > 1) g[rhs] = b;
  }
  template <int R, bool INV> static __device__ __forceinline__ void fft(V* v) { pk::dft<R, INV>(v); }
  template <bool CONJ> static __device__ __forceinline__ V tw(V v, const float2* p) {
    const float2 w = ldg_c(p);
    const pk::u64 c = pk::dup(w.x), s = pk::dup(w.y);
    return CONJ ? pk::tw_mulc(v, c, s) : pk::tw_mul(v, c, s);
  }
};

// Stage 0 < s < last, in place.
template <class P, bool PAIR, int NT, int s, bool INV>
__device__ __forceinline__ void stage(typename El<PAIR>::E* sm, const float2* __restrict__ tw, int tid, int nthr) {
  using X = El<PAIR>;
  constexpr int R = P::rad[s], M = P::M(s), Ls = M * R, B = P::N / R, off = Lay<P>::off(s);
  for (int t = tid; t < NT * 3 * B; t += nthr) {
    const int j = t / B, u = t - j * B, b = u / M, n1 = u - b * M;
    typename X::E* p = sm + j * Lay<P>::LW + Lay<P>::addr(b * Ls + n1);
    const float2* tws = tw + P::TWO(s) + n1;
    typename X::V v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = X::get(p + i * off);
    if (INV)
#pragma unroll
      for (int k = 1; k < R; ++k) v[k] = X::template tw<true>(v[k], tws + (k - 1) * M);
    X::template fft<R, INV>(v);
    if (!INV)
#pragma unroll
      for (int k = 1; k < R; ++k) v[k] = X::template tw<false>(v[k], tws + (k - 1) * M);
#pragma unroll
    for (int i = 0; i < R; ++i) X::put(p + i * off, v[i]);
  }
  __syncthreads();
}
template <class P, bool PAIR, int NT, int s, bool INV>
__device__ __forceinline__ void inner(typename El<PAIR>::E* sm, const float2* tw, int tid, int nthr) {
  if constexpr (s > 0 && s < P::nst - 1) {
    stage<P, PAIR, NT, s, INV>(sm, tw, tid, nthr);
    inner<P, PAIR, NT, INV ? s - 1 : s + 1, INV>(sm, tw, tid, nthr);
  }
}

template <class P, bool PAIR, int NT>
__global__ void __launch_bounds__(threads<P, PAIR>(NT), std::max(1, sm_threads<P, PAIR>() / threads<P, PAIR>(NT)))
k_pass_c(float2* __restrict__ t2, int L, int nlines, int nz, int nzp, const float2* __restrict__ tw,
         const float2* __restrict__ ghat, const int* done) {
  using X = El<PAIR>;
  constexpr int nthr = threads<P, PAIR>(NT);
  constexpr int N = P::N, LW = Lay<P>::LW;
  pdl_begin();
  if (done && *(volatile const int*)done) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Task* tk = reinterpret_cast<Task*>(smem_raw);
  typename X::E* lines = reinterpret_cast<typename X::E*>(smem_raw + NT * sizeof(Task));
  const int tid = threadIdx.x;
  const size_t fstride = (size_t)nlines * nzp;  // between fields
  if (tid < NT) {
    const int per = PAIR ? (L + 1) / 2 : L;     // tasks of a line
    const long long task = (long long)blockIdx.x * NT + tid;
    const long long line = task / per;
    const int l = (int)(task - line * per) * (PAIR ? 2 : 1);
    Task t{0, 0, 0, 0};
    if (line < nlines) {
      t.src = (long long)(3 * l * fstride) + line * nzp;
      t.gl = line * 6 * N;
      t.n = PAIR && l + 1 < L ? 2 : 1;
      t.rhs = t.n == 2 ? (long long)(3 * fstride) : 0;
    }
    tk[tid] = t;
  }
  __syncthreads();
  {  // first stage: T2 -> shared memory (rows past nz are zero padding; at least half of every butterfly)
    constexpr int R = P::rad[0], M = P::M(0), off = Lay<P>::off(0);
    for (int t = tid; t < NT * 3 * M; t += nthr) {
      const int j = t / M, n1 = t - j * M, k = j / 3, c = j - 3 * k;
      if (tk[k].n == 0) continue;
      const float2* g = t2 + tk[k].src + c * fstride + n1;
      const long long rhs = tk[k].rhs;
      typename X::V v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = (2 * i < R && n1 + i * M < nz) ? X::load(g + i * M, rhs) : X::zero();
      X::template fft<R, false>(v);
#pragma unroll
      for (int i = 1; i < R; ++i) v[i] = X::template tw<false>(v[i], tw + (i - 1) * M + n1);
      typename X::E* p = lines + j * LW + Lay<P>::addr(n1);
#pragma unroll
      for (int i = 0; i < R; ++i) X::put(p + i * off, v[i]);
    }
  }
  __syncthreads();
  inner<P, PAIR, NT, 1, false>(lines, tw, tid, nthr);
  {  // last forward stage, Green product, first inverse stage (no twiddles)
    constexpr int R = P::Rl, B = N / R, H = PAIR ? 2 : 1;
    float2* const l2 = reinterpret_cast<float2*>(lines);
    for (int t = tid; t < NT * B * H; t += nthr) {
      const int h = t % H, u = t / H, k = u / B, b = u - k * B;
      if (h >= tk[k].n) continue;
      float2* p = l2 + (3 * k * LW + b * Lay<P>::S) * H + h;
      const float2* gl = ghat + tk[k].gl + b;
      float2 e0[R], e1[R], e2[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        e0[i] = p[i * H];
        e1[i] = p[(LW + i) * H];
        e2[i] = p[(2 * LW + i) * H];
      }
      dft<R, false>(e0);
      dft<R, false>(e1);
      dft<R, false>(e2);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float2* g = gl + i * B;
        const float2 gxx = ldg_c(g), gxy = ldg_c(g + N), gxz = ldg_c(g + 2 * N);
        const float2 gyy = ldg_c(g + 3 * N), gyz = ldg_c(g + 4 * N), gzz = ldg_c(g + 5 * N);
        const float2 x = e0[i], y = e1[i], z = e2[i];
        e0[i] = cadd(cadd(cmul(gxx, x), cmul(gxy, y)), cmul(gxz, z));
        e1[i] = cadd(cadd(cmul(gxy, x), cmul(gyy, y)), cmul(gyz, z));
        e2[i] = cadd(cadd(cmul(gxz, x), cmul(gyz, y)), cmul(gzz, z));
      }
      dft<R, true>(e0);
      dft<R, true>(e1);
      dft<R, true>(e2);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        p[i * H] = e0[i];
        p[(LW + i) * H] = e1[i];
        p[(2 * LW + i) * H] = e2[i];
      }
    }
  }
  __syncthreads();
  inner<P, PAIR, NT, P::nst - 2, true>(lines, tw, tid, nthr);
  {  // last inverse stage: shared memory -> T2 (rows past nz dropped)
    constexpr int R = P::rad[0], M = P::M(0), off = Lay<P>::off(0);
    for (int t = tid; t < NT * 3 * M; t += nthr) {
      const int j = t / M, n1 = t - j * M, k = j / 3, c = j - 3 * k;
      if (tk[k].n == 0) continue;
      const typename X::E* p = lines + j * LW + Lay<P>::addr(n1);
      typename X::V v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = X::get(p + i * off);
#pragma unroll
      for (int i = 1; i < R; ++i) v[i] = X::template tw<true>(v[i], tw + (i - 1) * M + n1);
      X::template fft<R, true>(v);
      float2* g = t2 + tk[k].src + c * fstride + n1;
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (2 * i < R && n1 + i * M < nz) X::store(g + i * M, tk[k].rhs, tk[k].n, v[i]);
    }
  }
}

template <class P, bool PAIR, int NT>
cudaError_t launch_nt(const MvpGeom& g, float2* t2, int L, const float2* tw, const float2* ghat, long long ntask,
                      cudaStream_t st, const int* done) {
  constexpr int smem = smem_bytes<P, PAIR>(NT);
  static std::once_flag once;
  static cudaError_t cfg = cudaSuccess;
  std::call_once(once, [] {
    cfg = cudaFuncSetAttribute(k_pass_c<P, PAIR, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  if (cfg != cudaSuccess) return cfg;
  launch_pdl(k_pass_c<P, PAIR, NT>, (unsigned)((ntask + NT - 1) / NT), threads<P, PAIR>(NT), smem, st, t2, L, g.Px * g.Py, g.nz,
             g.nzp, tw, ghat, done);
  return cudaGetLastError();
}

template <class P, bool PAIR>
cudaError_t launch(const MvpGeom& g, float2* t2, int L, const float2* tw, const float2* ghat, cudaStream_t st,
                   const int* done) {
  const long long ntask = (long long)g.Px * g.Py * (PAIR ? (L + 1) / 2 : L);
  return launch_nt<P, PAIR, tasks<P, PAIR>()>(g, t2, L, tw, ghat, ntask, st, done);
}

// Runs pass C when the length is in range and f = 3.  MvpTune::zkern 1 runs pairs, 0 does not; by default pairs for even
// L and from L = 7: an empty half costs less than the pairs save there (9216 lines of 150, per right-hand side: pairs
// 12.8 us at L = 16, single 13.9; at L = 3 19.0 and 16.4).
template <class P>
bool launch(const MvpGeom& g, float2* t2, int L, const float2* tw, const float2* ghat, cudaStream_t st, const int* done,
            cudaError_t* err) {
  if constexpr (supported<P>()) {
    if (g.f != 3) return false;
    using Q = typename Own<P>::type;
    const bool pair = g.tune.zkern < 0 ? L % 2 == 0 || L >= 7 : g.tune.zkern == 1;
    *err = pair ? launch<Q, true>(g, t2, L, tw, ghat, st, done) : launch<Q, false>(g, t2, L, tw, ghat, st, done);
    return true;
  }
  return false;
}

}  // namespace zcol
}  // namespace bdda
