// Block MVP of the FP64 and double-float precisions on the 64-bit fixed-point
// FFT core (fx_fft.cuh): the same five passes A-E as the complex FP32 MVP
// (mvp_launch.cuh).
//
// T1 / T2 hold fixed-point values (2 x 64 bits per element, the size of complex
// FP64) in lines of the pass that wrote them, each line shifted up to 62 bits
// with an exponent in a side array (FxExps):
//   pass A -> ea[f][y][z] (x lines), B -> eb[f][x][z] (y lines), C -> ec[f][x][y]
//   (z lines), D -> eb again.
// The next pass aligns the elements of its lines, which come from lines of
// different exponents, to the largest one: two 64-bit shifts and an addition
// per part, where a conversion to FP64 and back took 80 instructions per
// element (64-bit adds and shifts run at 32 per clock and SM).  Only pass A
// converts from FP64 (the gathered sites) and pass E to FP64 (the scattered
// ones), so the values between the passes carry more bits than FP64's 53.
//
// The Green spectrum is held as Q62 integers with one exponent per (x, y) line
// and component.  In pass C every component of the vectors and of the product
// has an exponent of its own too: where components do not couple (the normal
// one of a flat target, the axial one of a chain; magnetic and electric ones at
// small k d) a small one keeps its bits beside a large one.  The terms of a row
// are aligned to its largest term as they are multiplied.
//
// The two precisions differ only in the vectors' storage (Io64, IoDf): pass E
// adds diag o x and scales by jpre in FP64 on the occupied sites (3% of a
// line's points in a typical aggregate).
//
// CTAs of the strided passes hold 8 z-columns (128-byte rows), four warps with
// two lines each, one tile per CTA: 4-6 such CTAs share an SM, so one's copies
// overlap another's arithmetic.
#include <algorithm>
#include <mutex>

#include "fx_fft.cuh"
#include "mvp.hpp"
#include "pdl.cuh"
#include "tile_passes.cuh"

namespace bdda {

namespace {

using fx::Acc;
using fx::Fac;
using fx::Split;
using fx::Val;

constexpr int kFxWarps = 4;                    // warps of a strided pass's CTA
constexpr int kFxThreads = kFxWarps * 32;
constexpr int kFxLines = kTZ / kFxWarps;       // lines per warp
constexpr int kFxRows = kFxThreads / kTZ;      // rows a tile copy moves at once

// CTAs per SM the kernels are compiled for: registers against resident warps.
// Measured at one CTA fewer / more: y passes N=16384, L=16 (Py=160) 1.97 /
// 1.89 ms for both, N=65536, L=16 (Py=270, 43 KB of lines per CTA) 10.5 /
// 10.9 ms; pass C 4.39 / 3.89 (Pz=150) and 20.4 / 20.9 ms (Pz=250, where only
// two CTAs fit).  So the larger count where that many fit in shared memory.
constexpr int kXMany = 6, kXFew = 5;  // passes A, B, D, E
constexpr int kCMany = 3, kCFew = 2;  // pass C, f = 3
constexpr int kCSix = 2;              // pass C, f = 6
constexpr int kSmemPerSm = 228 * 1024, kSmemReserved = 1024;  // shared memory of an SM, and what each CTA takes of it beside its own
bool fits(int ctas, int smem) { return ctas * (smem + kSmemReserved) <= kSmemPerSm; }

__device__ __forceinline__ bool skip(const int* done) { return done && *(volatile const int*)done; }
__device__ __forceinline__ int clog2(int n) { return n <= 1 ? 0 : 32 - __clz(n - 1); }
__device__ __forceinline__ Val raw(double2 v) { return {__double_as_longlong(v.x), __double_as_longlong(v.y)}; }

// Vector storage: complex FP64, or double-float pairs (exact sums in FP64 on read).
struct Io64 {
  using E = double2;
  static __device__ __forceinline__ double2 load(const E* p) { return *p; }
  static __device__ __forceinline__ void store(E* p, double2 v) { *p = v; }
};
struct IoDf {
  using E = dfc;
  static __device__ __forceinline__ double2 load(const E* p) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    return make_double2((double)v.x + (double)v.y, (double)v.z + (double)v.w);
  }
  static __device__ __forceinline__ void store(E* p, double2 v) {
    const float hx = (float)v.x, hy = (float)v.y;
    // a value beyond FP32's range has no low part (inf - inf is not one)
    const float lx = isfinite(hx) ? (float)(v.x - (double)hx) : 0.f, ly = isfinite(hy) ? (float)(v.y - (double)hy) : 0.f;
    *reinterpret_cast<float4*>(p) = make_float4(hx, lx, hy, ly);
  }
};

// Scale of this warp's line (FP64 bits at line[addr(i)], i < n, element i written by lane i % 32): its largest value and
// the sum of its parts bound every value of its transform.  A line of tiny values is rewritten, each element by its lane: a
// __syncwarp() comes before others read it.
__device__ __forceinline__ fx::Scale line_scale(Val* line, const fx::Plan& p, int lane, int n) {
  auto largest = [&] {
    int k = 0;
    for (int i = lane; i < n; i += 32) {
      const Val v = line[p.addr(i)];
      k = max(k, max(fx::key(v.x), fx::key(v.y)));
    }
    return (int)__reduce_max_sync(0xffffffffu, (unsigned)k);
  };
  int k = largest();
  const bool tiny = fx::tiny(k);
  if (tiny) {
    for (int i = lane; i < n; i += 32) line[p.addr(i)] = fx::lift_tiny(line[p.addr(i)]);
    k = largest();
  }
  unsigned sum = 0;
  for (int i = lane; i < n; i += 32) {
    const Val v = line[p.addr(i)];
    sum += fx::sum_unit(v.x, k >> 20) + fx::sum_unit(v.y, k >> 20);
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  fx::Scale s = fx::make_scale(k, p.headroom(false, fx::sum_head(sum, n)));
  if (tiny) s.ebase -= 200;
  return s;
}

// Exponents and shifts of this warp's output lines (columns z ..), from their bits in use and the exponents eo of
// their values (kBadExp, kZeroExp kept): shs[j] for the drain, eg[z + j] for the next pass.
__device__ __forceinline__ void put_exps(const int* used, const int* eo, int lane, int* shs, int* eg, int z, int nz) {
#pragma unroll
  for (int j = 0; j < kFxLines; ++j) {
    const int s = fx::store_shift((int)__reduce_or_sync(0xffffffffu, (unsigned)used[j]));
    if (lane == 0) {
      shs[j] = s;
      if (z + j < nz) eg[z + j] = eo[j] == fx::kBadExp || eo[j] == fx::kZeroExp ? eo[j] : eo[j] - s;
    }
  }
}
__device__ __forceinline__ Val lift(Val v, int s) { return {fx::shl(v.x, s), fx::shl(v.y, s)}; }

// Alignment of this warp's lines, whose elements have the exponents ex[j exs + i], i < n: rsh for the first stage,
// eo the exponents of the transform's output.  Values are shifted right by what their own bits in use leave of the
// transform's headroom: a line's elements are usually well below the peaks of the lines they were stored in.
__device__ __forceinline__ void line_aligns(const Val* wl, const fx::Plan& p, const int* ex, int exs, int lane, int n, bool inv,
                                            int* rsh, int* eo) {
#pragma unroll
  for (int j = 0; j < kFxLines; ++j) {
    int e = fx::kZeroExp, cnt = 0;
    for (int i = lane; i < n; i += 32) {
      const int v = ex[j * exs + i];
      e = max(e, v);
      cnt += v > fx::kZeroExp;
    }
    e = __reduce_max_sync(0xffffffffu, e);
    cnt = (int)__reduce_add_sync(0xffffffffu, (unsigned)cnt);
    int used = 0;
    for (int i = lane; i < n; i += 32) used |= fx::bits_of(wl[j * p.LW + p.addr(i)]) >> min(e - ex[j * exs + i], 31);
    const int s = fx::fit_shift((int)__reduce_or_sync(0xffffffffu, (unsigned)used), p.headroom(inv, clog2(cnt)));
    rsh[j] = e + s;
    eo[j] = e == fx::kBadExp || e == fx::kZeroExp ? e : e + s + p.D;
  }
}

// Fill of a tile: rows of 8 columns, one 16-byte copy per element (zero-filled where not valid).
template <class Valid>
__device__ __forceinline__ void fill_tile(Val* lines, const fx::Plan& p, const void* srcv, size_t stride, int nrows, int col,
                                          int row, Valid valid) {
  Val* lb = lines + col * p.LW;
  const Val* src = static_cast<const Val*>(srcv);
  const Val* g = src + (size_t)row * stride;
  for (int r = row; r < nrows; r += kFxRows, g += kFxRows * stride) {
    const bool ok = valid(r);
    tile::cp_async<16>(lb + p.addr(r), ok ? g : src, ok);
  }
  tile::cp_commit();
  tile::cp_wait<0>();
  __syncthreads();
}

// ---------------------------------------------------------------- pass A
template <class Io, int MB>
__global__ void __launch_bounds__(kFxThreads, MB)
k_fx_a(const typename Io::E* __restrict__ x, int ldx, int nfield, int fpg, int fc, const int* __restrict__ occ,
       const int* __restrict__ tiles, int nx, int ny, int nz, int nzp, int nzt, fx::Plan p, const Fac* __restrict__ tw,
       Val* __restrict__ t1, int* __restrict__ ea, const int* done) {
  pdl_begin();
  if (skip(done)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Val* lines = reinterpret_cast<Val*>(smem_raw);                 // [kTZ][LW]
  int* socc = reinterpret_cast<int*>(lines + kTZ * p.LW);        // [nx][kTZ]
  int* shs = socc + nx * kTZ;                                    // [kTZ] shift of each line's output
  const int tile = tiles[blockIdx.x];
  const int y = tile / nzt, z0 = (tile - y * nzt) * kTZ;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int idx = tid; idx < nx * kTZ; idx += kFxThreads) {
    const int xi = idx >> 3, z = z0 + (idx & 7);
    socc[idx] = z < nz ? occ[((size_t)xi * ny + y) * nz + z] : -1;
  }
  __syncthreads();
  const size_t rowstride = (size_t)ny * nzp;
  const int col = tid & (kTZ - 1), row = tid / kTZ;
  const int f0 = blockIdx.y * fpg, fend = min(nfield, f0 + fpg);
  for (int f = f0; f < fend; ++f) {
    const int l = f / fc, c = f - l * fc;
    const typename Io::E* xc = x + (size_t)l * ldx + c;
    Val* wl = lines + kFxLines * warp * p.LW;
    int rsh[kFxLines], eo[kFxLines], used[kFxLines] = {};
#pragma unroll
    for (int j = 0; j < kFxLines; ++j) {
      for (int xi = lane; xi < nx; xi += 32) {
        const int m = socc[xi * kTZ + kFxLines * warp + j];
        wl[j * p.LW + p.addr(xi)] = m >= 0 ? raw(Io::load(xc + fc * (size_t)m)) : Val{0, 0};
      }
      const fx::Scale s = line_scale(wl + j * p.LW, p, lane, nx);
      rsh[j] = s.rsh0;
      eo[j] = s.bad ? fx::kBadExp : s.zero ? fx::kZeroExp : s.ebase + p.D;
    }
    __syncwarp();
    fx::forward<kFxLines, fx::kRaw, true, true>(wl, p, tw, lane, 32, nx, {rsh, nullptr, 0}, used);
    put_exps(used, eo, lane, shs + kFxLines * warp, ea + ((size_t)f * ny + y) * nzp, z0 + kFxLines * warp, nz);
    __syncthreads();
    if (z0 + col < nz) {
      const Val* lb = lines + col * p.LW;
      const int s = shs[col];
      Val* out = t1 + (size_t)f * p.N * rowstride + (size_t)y * nzp + z0 + col + (size_t)row * rowstride;
      for (int q = row; q < p.N; q += kFxRows, out += kFxRows * rowstride) *out = lift(lb[p.addr(q)], s);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- pass B / D
template <bool INV, int MB>
__global__ void __launch_bounds__(kFxThreads, MB)
k_fx_y(const Val* __restrict__ src, Val* __restrict__ dst, const unsigned char* __restrict__ tmask, int Px, int ny, int nz, int nzp,
       int nzt, fx::Plan p, const Fac* __restrict__ tw, const int* __restrict__ ein, int* __restrict__ eout,
       const int* done) {
  pdl_begin();
  if (skip(done)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Val* lines = reinterpret_cast<Val*>(smem_raw);          // [kTZ][LW]
  int* shs = reinterpret_cast<int*>(lines + kTZ * p.LW);  // [kTZ] shift of each line's output
  int* ex = shs + kTZ;                                    // element exponents: [kTZ][ny] forward, [Py] inverse
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int col = tid & (kTZ - 1), row = tid / kTZ;
  const int nin = INV ? p.N : ny, nout = INV ? ny : p.N;
  const int zt = blockIdx.x % nzt, z0 = zt * kTZ;
  const int r = blockIdx.x / nzt;  // f * Px + q
  const bool zval = z0 + col < nz;
  const int* ei = INV ? ein + (size_t)r * p.N : ein + (size_t)(r / Px) * ny * nzp + z0 + (zval ? col : 0);
  if constexpr (INV)
    for (int i = tid; i < nin; i += kFxThreads) ex[i] = ei[i];
  fill_tile(lines, p, src + (size_t)r * nin * nzp + z0 + (zval ? col : 0), nzp, nin, col, row, [&](int yy) {
    const bool ok = zval && (INV || tmask[(size_t)yy * nzt + zt]);
    if constexpr (!INV) ex[col * ny + yy] = ok ? ei[(size_t)yy * nzp] : fx::kZeroExp;
    return ok;
  });
  Val* wl = lines + kFxLines * warp * p.LW;
  const int exs = INV ? 0 : ny;
  const int* wex = INV ? ex : ex + kFxLines * warp * ny;
  int rsh[kFxLines], eo[kFxLines], used[kFxLines] = {};
  line_aligns(wl, p, wex, exs, lane, nin, INV, rsh, eo);
  if (!INV) fx::forward<kFxLines, fx::kAlign, true, true>(wl, p, tw, lane, 32, ny, {rsh, wex, exs}, used);
  else fx::inverse<kFxLines, fx::kAlign, true>(wl, p, tw, lane, 32, ny, {rsh, wex, exs}, used);
  put_exps(used, eo, lane, shs + kFxLines * warp, eout + (size_t)r * nzp, z0 + kFxLines * warp, nz);
  __syncthreads();
  if (!zval) return;
  const Val* lb = lines + col * p.LW;
  const int s = shs[col];
  Val* out = dst + (size_t)r * nout * nzp + z0 + col + (size_t)row * nzp;
  for (int yy = row; yy < nout; yy += kFxRows, out += (size_t)kFxRows * nzp)
    if (!INV || tmask[(size_t)yy * nzt + zt]) *out = lift(lb[p.addr(yy)], s);
}

// ---------------------------------------------------------------- pass E
template <class Io, int MB>
__global__ void __launch_bounds__(kFxThreads, MB)
k_fx_e(const Val* __restrict__ t1, const int* __restrict__ ein, int nfield, int fpg, int fc, const int* __restrict__ occ,
       const int* __restrict__ tiles, int nx, int ny, int nz, int nzp, int nzt, fx::Plan p, const Fac* __restrict__ tw,
       const typename Io::E* __restrict__ x, int ldx, const typename Io::E* __restrict__ diag,
       const typename Io::E* __restrict__ jpre, typename Io::E* __restrict__ y, int ldy, const int* done) {
  pdl_begin();
  if (skip(done)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Val* lines = reinterpret_cast<Val*>(smem_raw);           // [kTZ][LW]
  int* socc = reinterpret_cast<int*>(lines + kTZ * p.LW);  // [nx][kTZ]
  int* ex = socc + nx * kTZ;                               // [kTZ][Px] element exponents
  const int tile = tiles[blockIdx.x];
  const int yy = tile / nzt, z0 = (tile - yy * nzt) * kTZ;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int idx = tid; idx < nx * kTZ; idx += kFxThreads) {
    const int xi = idx >> 3, z = z0 + (idx & 7);
    socc[idx] = z < nz ? occ[((size_t)xi * ny + yy) * nz + z] : -1;
  }
  const size_t rowstride = (size_t)ny * nzp;
  const int col = tid & (kTZ - 1), row = tid / kTZ;
  const bool zval = z0 + col < nz;
  const int f0 = blockIdx.y * fpg, fend = min(nfield, f0 + fpg);
  for (int f = f0; f < fend; ++f) {
    const int l = f / fc, c = f - l * fc;
    const int* ei = ein + (size_t)f * p.N * nzp + z0 + (zval ? col : 0);
    fill_tile(lines, p, t1 + (size_t)f * p.N * rowstride + (size_t)yy * nzp + z0 + (zval ? col : 0), rowstride, p.N, col, row,
              [&](int q) {
                ex[col * p.N + q] = zval ? ei[(size_t)q * nzp] : fx::kZeroExp;
                return zval;
              });
    Val* wl = lines + kFxLines * warp * p.LW;
    const int* wex = ex + kFxLines * warp * p.N;
    int rsh[kFxLines], eo[kFxLines], used[kFxLines];
    line_aligns(wl, p, wex, p.N, lane, p.N, true, rsh, eo);
    fx::inverse<kFxLines, fx::kAlign, false>(wl, p, tw, lane, 32, nx, {rsh, wex, p.N}, used);
    for (int t = lane; t < kFxLines * nx; t += 32) {
      const int xi = t / kFxLines, j = t - xi * kFxLines;
      const int m = socc[xi * kTZ + kFxLines * warp + j];
      if (m < 0) continue;
      const size_t r = fc * (size_t)m + c;
      const int e = j ? eo[1] : eo[0];
      const Val b = fx::to_bits(wl[j * p.LW + p.addr(xi)], e, e == fx::kBadExp);
      double2 v = make_double2(__longlong_as_double(b.x), __longlong_as_double(b.y));
      if (diag != nullptr) v = cadd(v, cmul(Io::load(diag + r), Io::load(x + (size_t)l * ldx + r)));
      if (jpre != nullptr) v = cmul(v, Io::load(jpre + r));
      Io::store(y + (size_t)l * ldy + r, v);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- pass C
// v[3 h + c]
template <int N> __device__ __forceinline__ int half(const int (&v)[N], int h, int c) { return N == 6 && h ? v[N - 3 + c] : v[c]; }

// One warp per (x = q, y = qy, rhs l): fc component lines, blockDim.x / 32 warps per CTA.  Bound by the integer multiplier
// and the instructions around it.  An exponent per component costs the alignment of nine (f = 6: 30) factors per
// frequency: 1.84 -> 2.00 ms at Pz=120 (N=8192, L=16), 3.90 -> 4.20 at 150, f = 6 0.151 -> 0.175 at 54 (N=1200, L=4),
// against one for all of them, whose small components lost the bits between.  One shift for the rows of lines whose
// spectrum components are close was no faster (4.2 ms): the second product loop cost what it saved.
template <bool SIX, int MB>
__global__ void __launch_bounds__(kZWarps * 32, MB)
k_fx_c(Val* __restrict__ t2, int L, int Px, int Py, int nz, int nzp, fx::Plan p, const Fac* __restrict__ tw,
       const Fac* __restrict__ ghat, const int* __restrict__ gexp, const int* __restrict__ ein, int* __restrict__ eout,
       const int* done) {
  constexpr int fc = SIX ? 6 : 3, nc = SIX ? 9 : 6;
  pdl_begin();
  if (skip(done)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long task = (long long)blockIdx.x * (blockDim.x >> 5) + warp;
  if (task >= (long long)Px * Py * L) return;
  const int l = (int)(task % L);
  const int line = (int)(task / L);  // q * Py + qy
  const int Pz = p.N, LW = p.LW;
  Val* s0 = reinterpret_cast<Val*>(smem_raw) + (size_t)warp * fc * LW;
  const size_t fstride = (size_t)Px * Py * nzp, estride = (size_t)Px * nzp;
  Val* g0 = t2 + (size_t)(fc * l) * fstride + (size_t)line * nzp;
  const int* ei = ein + (size_t)(fc * l) * estride + (size_t)(line / Py) * nzp;
  int* eo = eout + (size_t)(fc * l) * Px * Py + line;
  const size_t eostride = (size_t)Px * Py;
  int em[fc];  // largest exponent of a component's elements
#pragma unroll
  for (int c = 0; c < fc; ++c) em[c] = fx::kZeroExp;
  for (int z = lane; z < nz; z += 32)
#pragma unroll
    for (int c = 0; c < fc; ++c) em[c] = max(em[c], ei[c * estride + z]);
  int emax = fx::kZeroExp;
#pragma unroll
  for (int c = 0; c < fc; ++c) {
    em[c] = __reduce_max_sync(0xffffffffu, em[c]);
    emax = max(emax, em[c]);
  }
  const int ge = lane < nc ? gexp[(size_t)line * nc + lane] : fx::kZeroExp;  // lane i: exponent of spectrum component i
  const bool gbad = __any_sync(0xffffffffu, ge == fx::kBadExp);
  if (emax <= fx::kZeroExp || emax == fx::kBadExp || gbad) {  // zero in, zero out; or not finite
    if (lane < fc) eo[lane * eostride] = gbad ? fx::kBadExp : emax;
    return;
  }
  int in[fc] = {};
  for (int z = lane; z < nz; z += 32) {
    const int a = p.addr(z);
#pragma unroll
    for (int c = 0; c < fc; ++c) {
      const Val v = fx::align(g0[c * fstride + z], em[c] + 1 - ei[c * estride + z]);
      in[c] |= fx::bits_of(v);
      s0[c * LW + a] = v;
    }
  }
  // each component to the forward transform's headroom; lane c keeps the exponent of component c's transform
  int fsh[fc], ev = fx::kZeroExp;
#pragma unroll
  for (int c = 0; c < fc; ++c) {
    fsh[c] = 64 - __clz(__reduce_or_sync(0xffffffffu, (unsigned)in[c])) - (fx::kTopBit - 1 - p.headroom(false, clog2(nz)));
    if (lane == c && em[c] > fx::kZeroExp) ev = em[c] + 1 + fsh[c] + p.D;
  }
  __syncwarp();
  constexpr int halves = SIX ? 2 : 1;
  // one copy of a transform's code for both halves: small launches wait for their instructions
#pragma unroll 1
  for (int h = 0; h < halves; ++h) {
    const int rsh[3] = {half(fsh, h, 0), half(fsh, h, 1), half(fsh, h, 2)};
    fx::forward<3, fx::kShift, true, false>(s0 + 3 * h * LW, p, tw, lane, 32, nz, {rsh, nullptr, 0}, nullptr);
  }
  // Lane 3 r + c: the terms of row r with component c of its own block of rows and, f = 6, of the other one.  All lanes of a
  // row: the exponent of its products, from its largest term (exponents of spectrum component and value).  Lane 3 r: the
  // shifts of its terms' values, byte c (a zero component's does not matter).
  const int tr = lane < 3 * fc ? lane / 3 : 0, tc = lane % 3, ta = tr % 3;
  auto term = [&](int c, int i) {
    const int v = __shfl_sync(0xffffffffu, ev, c), g = __shfl_sync(0xffffffffu, ge, i < 0 ? 0 : i);
    return i >= 0 && v > fx::kZeroExp && g > fx::kZeroExp ? v + g : fx::kZeroExp;
  };
  const int own = term(tr - ta + tc, fx::green_a(ta, tc));
  const int oth = SIX ? term((tr < 3 ? 3 : 0) + tc, fx::green_b(ta, tc)) : fx::kZeroExp;
  int er = max(own, oth);
  er = max(er, max(__shfl_down_sync(0xffffffffu, er, 1), __shfl_down_sync(0xffffffffu, er, 2)));
  er = __shfl_sync(0xffffffffu, er, lane - tc);
  if (er > fx::kZeroExp) er += fx::kProductBits;
  auto shifts = [&](int e) {
    const unsigned s = (unsigned)min(max(er - e, 1), 62) << (8 * tc);
    return s | __shfl_down_sync(0xffffffffu, s, 1) | __shfl_down_sync(0xffffffffu, s, 2);
  };
  const unsigned so = shifts(own), st = SIX ? shifts(oth) : 0;
  unsigned sown[fc], soth[fc];
#pragma unroll
  for (int r = 0; r < fc; ++r) {
    sown[r] = __shfl_sync(0xffffffffu, so, 3 * r);
    soth[r] = SIX ? __shfl_sync(0xffffffffu, st, 3 * r) : 0;
  }
  const Fac* gl = ghat + (size_t)line * nc * Pz;
  int used[fc] = {};
  for (int f = lane; f < Pz; f += 32) {
    const int a = p.addr(f);
    Fac g[nc];
#pragma unroll
    for (int c = 0; c < nc; ++c) g[c] = fx::ldfac(gl + (size_t)c * Pz + f);
    Val e[3], w[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      e[c] = s0[c * LW + a];
      w[c] = SIX ? s0[(3 + c) * LW + a] : Val{0, 0};
    }
    // one copy of a block row's code: unrolled, an MVP of N=99, f = 6, L=1 took 40.0 us, with the loops 38.6
#pragma unroll 1
    for (int h = 0; h < halves; ++h) {
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        Acc acc;
        const unsigned q = SIX && h ? sown[fc - 3 + r] : sown[r];
#pragma unroll
        for (int c = 0; c < 3; ++c) acc.mad(g[fx::green_a(r, c)], fx::split(fx::align(e[c], (int)(q >> (8 * c) & 255u))));
        Val v;
        if constexpr (SIX) {  // E' = A E + B M, M' = A M - B E
          Acc t{0, 0, 0, 0};
          const unsigned u = h ? soth[fc - 3 + r] : soth[r];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const int i = fx::green_b(r, c);
            if (i < 0) continue;
            const Split s = fx::split(fx::align(w[c], (int)(u >> (8 * c) & 255u)));
            if (r > c) t.msub(g[i], s);
            else t.mad(g[i], s);
          }
          v = acc.get(t, h != 0);
        } else {
          v = acc.get();
        }
        const int b = fx::bits_of(v);
        used[r] |= SIX && h ? 0 : b;
        if constexpr (SIX) used[3 + r] |= h ? b : 0;
        s0[(3 * h + r) * LW + a] = v;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const Val t = e[c];
        e[c] = w[c];
        w[c] = t;
      }
    }
  }
  __syncwarp();
  // bring each row's largest part (below 2^bits; 2^32 where no high word is in use) to the inverse transform's headroom
  int ish[fc], s[fc] = {};
#pragma unroll
  for (int r = 0; r < fc; ++r)
    ish[r] = 64 - __clz(__reduce_or_sync(0xffffffffu, (unsigned)used[r])) - (fx::kTopBit - 1 - p.headroom(true, clog2(Pz)));
#pragma unroll 1
  for (int h = 0; h < halves; ++h) {
    const int rsh[3] = {half(ish, h, 0), half(ish, h, 1), half(ish, h, 2)};
    int ou[3] = {};
    fx::inverse<3, fx::kShift, true>(s0 + 3 * h * LW, p, tw, lane, 32, nz, {rsh, nullptr, 0}, ou);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int t = fx::store_shift((int)__reduce_or_sync(0xffffffffu, (unsigned)ou[c]));
      if (lane == 3 * (3 * h + c)) eo[(3 * h + c) * eostride] = er > fx::kZeroExp ? er + rsh[c] + p.D - t : fx::kZeroExp;
#pragma unroll
      for (int k = c; k < fc; k += 3) s[k] = k == 3 * h + c ? t : s[k];
    }
  }
  for (int z = lane; z < nz; z += 32) {
    const int a = p.addr(z);
#pragma unroll
    for (int c = 0; c < fc; ++c) g0[c * fstride + z] = lift(s0[c * LW + a], s[c]);
  }
}

// ---------------------------------------------------------------- Green spectrum
// Forward transform in place of contiguous lines (FP64), two per warp.
__global__ void __launch_bounds__(kFxThreads)
k_fx_contig(double2* __restrict__ data, size_t nlines, fx::Plan p, const Fac* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Val* wl = reinterpret_cast<Val*>(smem_raw) + kFxLines * warp * p.LW;
  const size_t line0 = ((size_t)blockIdx.x * kFxWarps + warp) * kFxLines;
  int rsh[kFxLines], eb[kFxLines];
#pragma unroll
  for (int j = 0; j < kFxLines; ++j) {
    const bool ok = line0 + j < nlines;
    const Val* d = reinterpret_cast<const Val*>(data) + (line0 + j) * p.N;
    for (int i = lane; i < p.N; i += 32) wl[j * p.LW + p.addr(i)] = ok ? d[i] : Val{0, 0};
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < kFxLines; ++j) {
    const fx::Scale s = line_scale(wl + j * p.LW, p, lane, p.N);
    rsh[j] = s.rsh0;
    eb[j] = s.bad ? fx::kBadExp : s.ebase + p.D;
  }
  __syncwarp();  // line_scale may have rewritten the lines
  fx::forward<kFxLines, fx::kRaw, false, false>(wl, p, tw, lane, 32, p.N, {rsh, nullptr, 0}, nullptr);
#pragma unroll
  for (int j = 0; j < kFxLines; ++j) {
    if (line0 + j >= nlines) break;
    Val* d = reinterpret_cast<Val*>(data) + (line0 + j) * p.N;
    for (int i = lane; i < p.N; i += 32) d[i] = fx::to_bits(wl[j * p.LW + p.addr(i)], eb[j], eb[j] == fx::kBadExp);
  }
}

// Forward transform in place along the middle index of data[A][N][cc], 8 columns per CTA.
__global__ void __launch_bounds__(kFxThreads)
k_fx_strided(double2* __restrict__ data, size_t cc, fx::Plan p, const Fac* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Val* lines = reinterpret_cast<Val*>(smem_raw);
  int* eb = reinterpret_cast<int*>(lines + kTZ * p.LW);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int col = tid & (kTZ - 1), row = tid / kTZ;
  const size_t c = (size_t)blockIdx.x * kTZ + col;
  const bool ok = c < cc;
  double2* base = data + (size_t)blockIdx.y * p.N * cc;
  fill_tile(lines, p, base + (ok ? c : 0), cc, p.N, col, row, [&](int) { return ok; });
  Val* wl = lines + kFxLines * warp * p.LW;
  int rsh[kFxLines];
#pragma unroll
  for (int j = 0; j < kFxLines; ++j) {
    const fx::Scale s = line_scale(wl + j * p.LW, p, lane, p.N);
    rsh[j] = s.rsh0;
    if (lane == 0) eb[kFxLines * warp + j] = s.bad ? fx::kBadExp : s.ebase + p.D;
  }
  __syncwarp();  // line_scale may have rewritten the lines
  fx::forward<kFxLines, fx::kRaw, false, false>(wl, p, tw, lane, 32, p.N, {rsh, nullptr, 0}, nullptr);
  __syncthreads();
  if (!ok) return;
  const Val* lb = lines + col * p.LW;
  const int e = eb[col];
  Val* out = reinterpret_cast<Val*>(base) + c + (size_t)row * cc;
  for (int i = row; i < p.N; i += kFxRows, out += kFxRows * cc) *out = fx::to_bits(lb[p.addr(i)], e, e == fx::kBadExp);
}

// g[comp][qx][qy][qz] * scale -> out[qx][qy][comp][qz] as Q62 over a power of
// two 2^gexp of the line and component that leaves its moduli kGreenBits below
// 1: one warp per (qx, qy) line.
template <int NC>
__global__ void __launch_bounds__(256)
k_fx_pack(const double2* __restrict__ g, Fac* __restrict__ out, int* __restrict__ gexp, size_t nline, int Pz, double scale) {
  const size_t line = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (line >= nline) return;
  const int lane = threadIdx.x & 31;
  const size_t ng = nline * Pz;
  const double2* gl = g + line * Pz;
  double m[NC] = {};  // largest modulus sum of a component
  bool bad = false;
  for (int q = lane; q < Pz; q += 32)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const double2 v = gl[(size_t)c * ng + q];
      const double a = fabs(v.x) + fabs(v.y);
      bad = bad || !isfinite(a);
      m[c] = fmax(m[c], a);
    }
  bad = __any_sync(0xffffffffu, bad);
  // lane c: component c's exponent, the factor to its integers and, where that is beyond FP64's range, the rest of it
  int e = fx::kZeroExp;
  double mul = 0.0, more = 1.0;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const unsigned h = (unsigned)__double2hiint(m[c]);
    const unsigned top = __reduce_max_sync(0xffffffffu, h);
    const unsigned lo = __reduce_max_sync(0xffffffffu, h == top ? (unsigned)__double2loint(m[c]) : 0u);
    if (lane == c) m[0] = __hiloint2double((int)top, (int)lo);
  }
  if (lane < NC && m[0] * scale > 0.0) {
    frexp(m[0] * scale, &e);  // below 2^e
    e += fx::kGreenBits;
    mul = ldexp(scale, min(62 - e, 1000));
    more = ldexp(1.0, max(62 - e - 1000, 0));
  }
  if (bad) mul = 0.0;
  if (lane < NC) gexp[line * NC + lane] = bad ? fx::kBadExp : e;
  const bool tiny = __any_sync(0xffffffffu, more != 1.0);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const double f = __shfl_sync(0xffffffffu, mul, c), f2 = __shfl_sync(0xffffffffu, more, c);
    for (int q = lane; q < Pz; q += 32) {
      const double2 v = gl[(size_t)c * ng + q];
      double x = v.x * f, y = v.y * f;
      if (tiny) { x *= f2; y *= f2; }
      const long long re = __double2ll_rn(x), im = __double2ll_rn(y);
      Fac w;
      fx::split(re, w.rh, w.rl);
      fx::split(im, w.ih, w.il);
      out[(line * NC + c) * Pz + q] = w;
    }
  }
}

// Shared memory of a strided pass: lines, shifts, ints (exponents, occupancy).
int fx_smem(const fx::Plan& p, int ints) { return kTZ * p.LW * (int)sizeof(Val) + kTZ * 4 + ints * 4; }

cudaError_t configure() {
  static std::once_flag once;
  static cudaError_t cfg = cudaSuccess;
  std::call_once(once, [] {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    auto set = [&](const void* k) {
      if (cfg == cudaSuccess) cfg = cudaFuncSetAttribute(k, attr, kZSmemMax);
    };
    set((const void*)k_fx_a<Io64, kXMany>);
    set((const void*)k_fx_a<IoDf, kXMany>);
    set((const void*)k_fx_a<Io64, kXFew>);
    set((const void*)k_fx_a<IoDf, kXFew>);
    set((const void*)k_fx_y<false, kXMany>);
    set((const void*)k_fx_y<true, kXMany>);
    set((const void*)k_fx_y<false, kXFew>);
    set((const void*)k_fx_y<true, kXFew>);
    set((const void*)k_fx_e<Io64, kXMany>);
    set((const void*)k_fx_e<IoDf, kXMany>);
    set((const void*)k_fx_e<Io64, kXFew>);
    set((const void*)k_fx_e<IoDf, kXFew>);
    set((const void*)k_fx_c<false, kCMany>);
    set((const void*)k_fx_c<false, kCFew>);
    set((const void*)k_fx_c<true, kCSix>);
    set((const void*)k_fx_contig);
    set((const void*)k_fx_strided);
  });
  return cfg;
}

int num_sms() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 1;
  }();
  return n;
}

template <class Io>
cudaError_t launch(const MvpGeom& g, const FxTables& t, const void* xv, int ldx, void* yv, int ldy, int L, const void* diagv,
                   const void* jprev, const FxWork& w, cudaStream_t st, KernelTimer* timer, const int* done) {
  using E = typename Io::E;
  cudaError_t e = configure();
  if (e != cudaSuccess) return e;
  if (g.ntiles == 0) return cudaSuccess;  // no dipoles
  const E *x = (const E*)xv, *diag = (const E*)diagv, *jpre = (const E*)jprev;
  E* y = (E*)yv;
  const fx::Plan &px = t.plan[0], &py = t.plan[1], &pz = t.plan[2];
  const int nfield = g.f * L;
  // x passes: fields split over CTAs for about 24 CTAs per SM (four to six are resident)
  const int want = std::max(1, std::min(nfield, (24 * num_sms() + g.ntiles - 1) / g.ntiles));
  const int fpg = (nfield + want - 1) / want;
  const dim3 xgrid(g.ntiles, (nfield + fpg - 1) / fpg);
  const unsigned ygrid = (unsigned)((size_t)nfield * g.Px * g.nzt);
  Val *t1 = (Val*)w.t1, *t2 = (Val*)w.t2;
  auto begin = [&](int id) { if (timer) timer->begin(id, st); };
  auto end = [&](int id) { if (timer) timer->end(id, st); };
  begin(kPassA64);
  const int asm_ = fx_smem(px, kTZ * g.nx), bsm = fx_smem(py, kTZ * g.ny), dsm = fx_smem(py, g.Py),
            esm = fx_smem(px, kTZ * (g.nx + g.Px));
  auto* ka = fits(kXMany, asm_) ? k_fx_a<Io, kXMany> : k_fx_a<Io, kXFew>;
  launch_pdl(ka, xgrid, kFxThreads, asm_, st, x, ldx, nfield, fpg, g.f, g.occ, g.tiles, g.nx, g.ny, g.nz,
                                                                 g.nzp, g.nzt, px, t.tw[0], t1, w.ea, done);
  end(kPassA64);
  begin(kPassB64);
  auto* kb = fits(kXMany, bsm) ? k_fx_y<false, kXMany> : k_fx_y<false, kXFew>;
  launch_pdl(kb, ygrid, kFxThreads, bsm, st, t1, t2, g.tmask, g.Px, g.ny, g.nz, g.nzp, g.nzt, py,
                                                                    t.tw[1], w.ea, w.eb, done);
  end(kPassB64);
  begin(kPassC64);
  {
    const int per_warp = g.f * pz.LW * (int)sizeof(Val);
    const int wpc = z_warps_per_cta(per_warp);
    const long long ntask = (long long)g.Px * g.Py * L;
    const unsigned grid = (unsigned)((ntask + wpc - 1) / wpc);
    auto* kc = g.f == 6 ? k_fx_c<true, kCSix> : fits(kCMany, wpc * per_warp) ? k_fx_c<false, kCMany> : k_fx_c<false, kCFew>;
    launch_pdl(kc, grid, wpc * 32, wpc * per_warp, st, t2, L, g.Px, g.Py, g.nz, g.nzp, pz, t.tw[2], t.ghat, t.gexp, w.eb, w.ec, done);
  }
  end(kPassC64);
  begin(kPassD64);
  auto* kd = fits(kXMany, dsm) ? k_fx_y<true, kXMany> : k_fx_y<true, kXFew>;
  launch_pdl(kd, ygrid, kFxThreads, dsm, st, t2, t1, g.tmask, g.Px, g.ny, g.nz, g.nzp, g.nzt, py, t.tw[1],
                                                             w.ec, w.eb, done);
  end(kPassD64);
  begin(kPassE64);
  auto* ke = fits(kXMany, esm) ? k_fx_e<Io, kXMany> : k_fx_e<Io, kXFew>;
  launch_pdl(ke, xgrid, kFxThreads, esm, st, t1, w.eb, nfield, fpg, g.f, g.occ, g.tiles, g.nx, g.ny,
                                                                          g.nz, g.nzp, g.nzt, px, t.tw[0], x, ldx, diag, jpre,
                                                                          y, ldy, done);
  end(kPassE64);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_block_mvp_fx(const MvpGeom& g, const FxTables& t, bool df, const void* x, int ldx, void* y, int ldy, int L,
                                const void* diag, const void* jpre, const FxWork& w, cudaStream_t st,
                                KernelTimer* timer, const int* done) {
  return df ? launch<IoDf>(g, t, x, ldx, y, ldy, L, diag, jpre, w, st, timer, done)
            : launch<Io64>(g, t, x, ldx, y, ldy, L, diag, jpre, w, st, timer, done);
}

cudaError_t fx_green_transform(double2* data, int nc, const FxTables& t, cudaStream_t st) {
  cudaError_t e = configure();
  if (e != cudaSuccess) return e;
  const fx::Plan &px = t.plan[0], &py = t.plan[1], &pz = t.plan[2];
  const size_t nlines = (size_t)nc * px.N * py.N;
  k_fx_contig<<<(unsigned)((nlines + kTZ - 1) / kTZ), kFxThreads, kTZ * pz.LW * (int)sizeof(Val), st>>>(data, nlines, pz, t.tw[2]);
  k_fx_strided<<<dim3((unsigned)((pz.N + kTZ - 1) / kTZ), nc * px.N), kFxThreads, fx_smem(py, 0), st>>>(data, (size_t)pz.N, py, t.tw[1]);
  const size_t cc = (size_t)py.N * pz.N;
  k_fx_strided<<<dim3((unsigned)((cc + kTZ - 1) / kTZ), nc), kFxThreads, fx_smem(px, 0), st>>>(data, cc, px, t.tw[0]);
  return cudaGetLastError();
}

cudaError_t fx_green_pack(const double2* data, int nc, const FxTables& t, fx::Fac* ghat, int* gexp, double scale, cudaStream_t st) {
  const size_t nline = (size_t)t.plan[0].N * t.plan[1].N;
  const unsigned grid = (unsigned)((nline + 7) / 8);
  if (nc == 9) k_fx_pack<9><<<grid, 256, 0, st>>>(data, ghat, gexp, nline, t.plan[2].N, scale);
  else k_fx_pack<6><<<grid, 256, 0, st>>>(data, ghat, gexp, nline, t.plan[2].N, scale);
  return cudaGetLastError();
}

}  // namespace bdda
