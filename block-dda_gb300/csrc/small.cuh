// Single-CTA complex L x L algebra for the block Krylov solvers (included by
// solver.cu only).  Matrices are column-major in shared memory, M[i + j*L].
// Every routine is called by all kSmallThreads threads of the CTA and ends
// with a barrier.
//
// Replaces Eigen's partialPivLu / fullPivLu solves
// (bl_krylov_mvp_fft/bl_cocg_rq_mvp_fft.cpp:56,66, bl_cocg_rq_jacobi_mvp_fft.cpp:63,73,
// bl_bicgstab_mvp_fft.cpp:58-59,93, bl_bicggr_mvp_fft.cpp:51,110) and the L x L
// part of qr_reduced (qr_reduced.cpp:9-31, here as the Cholesky factors of
// CholQR2), so a whole Krylov iteration runs without a host round trip.
//
// Two arithmetics, R: double (complex FP64, double2 matrices) for FP64
// solves, and dfl (double-float, dfc matrices, ~48-bit significand) for the
// mixed-precision inner solves, whose block vectors are FP32 -- GB300 issues
// FP32 at 64 times its FP64 rate.  Inputs (Gram partials) and the state slots
// in global memory stay complex FP64 either way.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "krylov_kernels.cuh"

namespace bdda {

constexpr int kSmallThreads = 256;

template <typename R> struct SmallMat;
template <> struct SmallMat<double> { using M = double2; };
template <> struct SmallMat<dfl> { using M = dfc; };

// ---- double-float reciprocal and square root --------------------------------
// The FP32 result refined by Newton steps whose residual is evaluated in
// double-float (Dekker 1971; Hida, Li and Bailey 2001, "Algorithms for
// quad-double precision floating point arithmetic").
__device__ __forceinline__ dfl df_recip(dfl b) {
  const float q = __frcp_rn(b.hi);
  // e = 1 - b q to about 2^-48 of 1 (the FMA of the leading part is exact but for its last rounding), then one Newton
  // step with its second-order term: q (1 + e + e^2)
  const float e = fmaf(-b.lo, q, fmaf(-b.hi, q, 1.0f));
  return df_quick_two_sum(q, q * fmaf(e, e, e));
}
__device__ __forceinline__ dfl df_sqrt(dfl a) {
  if (!(a.hi > 0.0f)) return dfl(sqrtf(a.hi), 0.0f);  // zero, negative or NaN: the FP32 answer
  const float x = sqrtf(a.hi);
  const dfl xx(x, 0.0f);
  return xx + dfl((a - xx * xx).hi * (0.5f / x), 0.0f);
}

// ---- scalar and complex helpers of the two arithmetics ---------------------
__device__ __forceinline__ double r_recip(double a) { return 1.0 / a; }
__device__ __forceinline__ dfl r_recip(dfl a) { return df_recip(a); }
__device__ __forceinline__ double r_sqrt(double a) { return sqrt(a); }
__device__ __forceinline__ dfl r_sqrt(dfl a) { return df_sqrt(a); }
__device__ __forceinline__ bool r_pos_finite(double a) { return a > 0.0 && isfinite(a); }
__device__ __forceinline__ bool r_pos_finite(dfl a) { return a.hi > 0.0f && isfinite(a.hi) && isfinite(a.lo); }
__device__ __forceinline__ double r_to_double(double a) { return a; }
__device__ __forceinline__ double r_to_double(dfl a);
template <typename R> __device__ __forceinline__ R r_const(float v) { return R(v); }
template <> __device__ __forceinline__ dfl r_const<dfl>(float v) { return dfl(v, 0.0f); }

__device__ __forceinline__ double2 m_to_double2(double2 a) { return a; }
// Double-float <-> FP64 with the values of dfl(v) and df_to_double(a), the conversions done on the bit patterns
// (conversion instructions and FP64 additions issue at two per clock and SM).
__device__ __forceinline__ dfl df_from_double(double v) {
  const int h = __double2hiint(v);
  const unsigned l = (unsigned)__double2loint(v);
  const int e = (h >> 20) & 0x7ff;
  if (e < 960 || e > 1140) return ((h << 1) | (int)l) == 0 ? dfl(0.0f, 0.0f) : dfl(v);
  const int up = (int)((l >> 28) & 1u);  // the leading part is rounded to nearest (a tie away from zero)
  const int r = (int)(l & 0x1fffffffu) - (up << 29);
  const unsigned hb = ((unsigned)(e - 896) << 23 | ((unsigned)h & 0xfffffu) << 3 | l >> 29) + (unsigned)up;
  const float lo = (float)r * __uint_as_float((unsigned)(e - 896 - 52) << 23);
  const unsigned sg = (unsigned)h & 0x80000000u;
  return dfl(__uint_as_float(hb | sg), __uint_as_float(__float_as_uint(lo) ^ sg));
}
__device__ __forceinline__ double d_from_float(float v) {
  const unsigned b = __float_as_uint(v);
  const unsigned e = (b >> 23) & 0xffu;
  if (e == 0 || e == 0xff) return (b << 1) == 0 ? __hiloint2double((int)b, 0) : (double)v;
  return __hiloint2double((int)((b & 0x80000000u) | ((e + 896) << 20) | ((b & 0x7fffffu) >> 3)), (int)(b << 29));
}
__device__ __forceinline__ double d_from_df(dfl a) { return d_from_float(a.hi) + d_from_float(a.lo); }
__device__ __forceinline__ double r_to_double(dfl a) { return d_from_df(a); }
__device__ __forceinline__ double2 m_to_double2(dfc a) { return make_double2(d_from_df(a.x), d_from_df(a.y)); }
template <typename M> __device__ M m_from_double2(double2 a);
template <> __device__ __forceinline__ double2 m_from_double2<double2>(double2 a) { return a; }
template <> __device__ __forceinline__ dfc m_from_double2<dfc>(double2 a) { return cmake(df_from_double(a.x), df_from_double(a.y)); }

template <typename M> __device__ __forceinline__ auto m_abs2(M a) { return a.x * a.x + a.y * a.y; }
template <typename M> __device__ __forceinline__ M m_neg(M a) { return cmake(-a.x, -a.y); }
template <typename M> __device__ __forceinline__ bool m_finite(M a) {
  return isfinite(r_to_double(a.x)) && isfinite(r_to_double(a.y));
}
// Whether 1 / a keeps FP64's precision (solves of very small or large right-hand sides have Gram sums near its ends).
__device__ __forceinline__ bool r_recip_ok(double a) { return a > 0x1p-1000 && a < 0x1p1000; }
__device__ __forceinline__ bool r_recip_ok(dfl) { return true; }
// 1 / b; operands are O(1) pivots (no scaling against overflow of |b|^2)
__device__ __forceinline__ double2 m_recip(double2 b) {
  const double n = b.x * b.x + b.y * b.y;
  if (!r_recip_ok(n)) return make_double2(b.x / n, -b.y / n);
  const double d = 1.0 / n;
  return make_double2(b.x * d, -b.y * d);
}
__device__ __forceinline__ dfc m_recip(dfc b) {
  const dfl d = df_recip(b.x * b.x + b.y * b.y);
  return cmake(b.x * d, -(b.y * d));
}
// conj(a) / b, b real
__device__ __forceinline__ double2 m_over(double2 a, double b) { return make_double2(a.x / b, -a.y / b); }
__device__ __forceinline__ dfc m_over(dfc a, dfl b) {
  const dfl q = df_recip(b);
  return cmake(a.x * q, -(a.y * q));
}
// complex FP64 helpers used outside the templated routines
__device__ __forceinline__ double cabs2(double2 a) { return a.x * a.x + a.y * a.y; }
// a / b, no scaling against overflow of |b|^2
__device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
  const double d = b.x * b.x + b.y * b.y;
  return make_double2((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}
__device__ __forceinline__ bool cfinite(double2 a) { return isfinite(a.x) && isfinite(a.y); }

// A Gram matrix as the row kernels leave it: n = 0: reduced, complex FP64 at p; else n partial matrices of type P (FP64 or
// double-float), `stride` elements apart.
struct GramRef {
  const void* p;
  int n, stride;
};
// dst = the matrix at element offset off.  Partials (LL <= 64, a separate reduction launch costs more than it saves there)
// are summed by S threads per entry and a fixed tree.
template <typename R, typename P>
__device__ void sm_gram(typename SmallMat<R>::M* dst, GramRef g, int off, int LL) {
  using M = typename SmallMat<R>::M;
  if (g.n == 0) {
    const double2* q = static_cast<const double2*>(g.p) + off;
    for (int e = threadIdx.x; e < LL; e += blockDim.x) dst[e] = m_from_double2<M>(__ldg(q + e));
    return;
  }
  __shared__ P red[kSmallThreads];
  const P* q = static_cast<const P*>(g.p) + off;
  const int sh = LL <= 1 ? 0 : 32 - __clz(LL - 1);
  const int e = threadIdx.x & ((1 << sh) - 1), s = threadIdx.x >> sh, S = kSmallThreads >> sh;
  P acc[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) gp_zero(acc[u]);
  if (e < LL) {
    int p = s;
    for (; p + 3 * S < g.n; p += 4 * S) {
      P v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = q[(size_t)(p + u * S) * g.stride + e];
#pragma unroll
      for (int u = 0; u < 4; ++u) gp_add(acc[u], v[u]);
    }
    for (; p < g.n; p += S) gp_add(acc[0], q[(size_t)p * g.stride + e]);
  }
  gp_add(acc[0], acc[1]);
  gp_add(acc[2], acc[3]);
  gp_add(acc[0], acc[2]);
  __syncthreads();  // red may still be read by a previous call's tree
  red[threadIdx.x] = acc[0];
  __syncthreads();
  for (int o = S >> 1; o > 0; o >>= 1) {
    if (s < o) gp_add(red[threadIdx.x], red[threadIdx.x + (o << sh)]);
    __syncthreads();
  }
  if (s == 0 && e < LL) {
    if constexpr (std::is_same<M, P>::value) dst[e] = red[e];
    else dst[e] = m_from_double2<M>(gp_d2(red[e]));
  }
}

// state slot (complex FP64, global) <-> shared matrix; no barrier: the caller has one before the other side is used
template <typename M> __device__ void sm_load(M* dst, const double2* src, int LL) {
  for (int e = threadIdx.x; e < LL; e += blockDim.x) dst[e] = m_from_double2<M>(src[e]);
}
template <typename M> __device__ void sm_store(double2* dst, const M* src, int LL, bool negate = false) {
  for (int e = threadIdx.x; e < LL; e += blockDim.x) dst[e] = m_to_double2(negate ? m_neg(src[e]) : src[e]);
}

// Element (i, j0 + s step) of an L-row matrix for thread `rank` of `size`: rows padded to a power of two, so that no
// index needs an integer division (a runtime division is as long as the arithmetic it would feed).
struct Cells {
  int i, j0, step;
  __device__ Cells(int rank, int size, int L) {
    const int sh = L <= 2 ? 1 : 32 - __clz(L - 1);
    i = rank & ((1 << sh) - 1);
    j0 = rank >> sh;
    step = size >> sh;
  }
};

// C = op(A) * B with op = transpose (TA=1) or identity (TA=0); C must not alias.
template <typename M> __device__ void sm_matmul(M* Cm, const M* A, const M* B, int L, bool TA) {
  const Cells c((int)threadIdx.x, (int)blockDim.x, L);
  if (c.i < L)
    for (int j = c.j0; j < L; j += c.step) {
      M s = czero<M>();
      for (int k = 0; k < L; ++k) s = cadd(s, cmul(TA ? A[k + c.i * L] : A[c.i + k * L], B[k + j * L]));
      Cm[c.i + j * L] = s;
    }
  __syncthreads();
}

// ---- teams --------------------------------------------------------------------
// The sequential L x L factorisations run on a team: the whole CTA (step
// phases separated by __syncthreads) or, for L <= kWarpL, warp 0 alone (phases
// separated by __syncwarp; the other warps wait at the routine's final
// barrier).  For small L a step's phase is a few elements per lane, so the
// CTA-wide barriers cost more than the work they separate (L = 2: 10% more
// solves per second at N=1024); at L = 16 one warp's share of the trailing
// updates (about 40 double-float elements per lane) outweighs the barriers.
constexpr int kWarpL = 8;
struct CtaTeam {
  int rank, size;
  __device__ void sync() const { __syncthreads(); }
};
struct WarpTeam {
  int rank, size;
  __device__ void sync() const { __syncwarp(); }
};

// Integer that orders values by |a|^2 (the top 32 bits of its FP64 or FP32 pattern; NaN is the largest), 0 only where
// |a|^2 is.
__device__ __forceinline__ unsigned mag_key(double2 a) {
  const double m = m_abs2(a);
  const unsigned h = (unsigned)__double2hiint(m);
  return h != 0 ? h : __double2loint(m) != 0 ? 1u : 0u;
}
__device__ __forceinline__ unsigned mag_key(dfc a) { return __float_as_uint(a.x.hi * a.x.hi + a.y.hi * a.y.hi); }

// Pivot of step k by one warp: the largest |a| (to the 20 or 23 bits of mag_key; the first in row order among equals, with
// full in column order first) of the rows and columns not used yet.  Lane r holds row r.  Where all of them are zero the
// pivot is one of these zeros (used columns keep old values), which the caller's test of it refuses.
template <typename M>
__device__ __forceinline__ void find_pivot(const M* A, int L, int k, bool full, unsigned rows, unsigned cols, int* pr, int* pc) {
  const int lane = threadIdx.x & 31;
  const bool row = lane < L && ((rows >> lane) & 1u);
  unsigned best = 0;
  int bc = full ? __ffs((int)cols) - 1 : k;
  if (!full) {
    best = row ? mag_key(A[lane + k * L]) : 0;
  } else if (row) {
    for (int c = 0; c < L; ++c)
      if ((cols >> c) & 1u) {
        const unsigned v = mag_key(A[lane + c * L]);
        if (v > best) { best = v; bc = c; }
      }
  }
  const unsigned mx = __reduce_max_sync(0xffffffffu, best);
  const unsigned at = row && best == mx ? (unsigned)(bc * 32 + lane) : 0xffffffffu;
  const unsigned w = __reduce_min_sync(0xffffffffu, at);
  *pr = (int)(w & 31u);
  *pc = full ? (int)((w >> 5) & 31u) : k;
}

// LU solve on a team (see sm_lu_solve); *bad (shared) set on a zero /
// non-finite pivot or result.  No rows or columns are moved: step k records the
// row and column it eliminates with (prow, pcol) and updates the rows not used
// yet.  A step is a chain -- pivot search, complex reciprocal, multiplier,
// update -- so what its length is made of is cut:
//  * in double-float, and on a single warp, every warp finds the pivot and
//    every thread takes the reciprocal and its row's multiplier itself, and a
//    step has one barrier (RED);
//  * FP64 issues two operations per clock and SM, so on the whole CTA one warp
//    does the search and the reciprocal and one thread per row the multiplier.
// With the factor and inverse of ldl_team and the state loaded in one trip, the L x L steps of a mixed solve of N=8192,
// L=16 went from 44.7 to 29.5 us per launch (event-timed).
template <typename R, bool RED, class Team>
__device__ void lu_solve_team(const Team tm, typename SmallMat<R>::M* A, typename SmallMat<R>::M* B, int L, int nrhs,
                              bool full, int* prow, typename SmallMat<R>::M* dinv, int* pcol, int* bad) {
  using M = typename SmallMat<R>::M;
  const Cells c(tm.rank, tm.size, L);
  unsigned rows = L == 32 ? 0xffffffffu : (1u << L) - 1u, cols = rows;
  const bool mine = c.i < L;
  tm.sync();
  for (int k = 0; k < L; ++k) {
    int pr = 0, pc = 0;
    M f;
    if constexpr (RED) {
      find_pivot(A, L, k, full, rows, cols, &pr, &pc);
      const M p = A[pr + pc * L];
      if (full) tm.sync();  // the search read columns this step updates
      if (!r_pos_finite(m_abs2(p))) { if (tm.rank == 0) *bad = 1; return; }
      const M pi = m_recip(p);
      if (tm.rank == 0) { prow[k] = pr; pcol[k] = pc; dinv[k] = pi; }
      if (mine) f = cmul(A[c.i + pc * L], pi);
    } else {
      if (tm.rank < 32) {
        find_pivot(A, L, k, full, rows, cols, &pr, &pc);
        const M p = A[pr + pc * L];
        const M pi = m_recip(p);
        if (tm.rank == 0) {
          prow[k] = pr; pcol[k] = pc; dinv[k] = pi;
          if (!r_pos_finite(m_abs2(p))) *bad = 1;
        }
        if (tm.rank < L && tm.rank != pr && ((rows >> tm.rank) & 1u)) A[tm.rank + pc * L] = cmul(A[tm.rank + pc * L], pi);
      }
      tm.sync();
      if (*bad) return;
      pr = prow[k]; pc = pcol[k];
      if (mine) f = A[c.i + pc * L];
    }
    rows &= ~(1u << pr);
    cols &= ~(1u << pc);
    if (mine && ((rows >> c.i) & 1u)) {
      for (int j = c.j0; j < L + nrhs; j += c.step) {
        if (j < L && !((cols >> j) & 1u)) continue;
        M* col = j < L ? A + j * L : B + (j - L) * L;
        col[c.i] = csub(col[c.i], cmul(f, col[pr]));
      }
    }
    tm.sync();
  }
  // back substitution: the unknown of step k is its pivot row's right-hand side over the pivot once the later ones have
  // been taken out; each step takes it out of the rows used before, one barrier a step
  for (int k = L - 1; k > 0; --k) {
    const int pr = prow[k], pc = pcol[k];
    rows |= 1u << pr;  // rows used at step k and after
    if (mine && !((rows >> c.i) & 1u)) {
      const M u = cmul(A[c.i + pc * L], dinv[k]);
      for (int j = c.j0; j < nrhs; j += c.step) {
        M* col = B + j * L;
        col[c.i] = csub(col[c.i], cmul(u, col[pr]));
      }
    }
    tm.sync();
  }
  // X[pcol[k]] = B[prow[k]] / pivot (through A, no longer needed)
  if (mine)
    for (int j = c.j0; j < nrhs; j += c.step) A[pcol[c.i] + j * L] = cmul(B[prow[c.i] + j * L], dinv[c.i]);
  tm.sync();
  if (mine)
    for (int j = c.j0; j < nrhs; j += c.step) {
      const M v = A[c.i + j * L];
      if (!m_finite(v)) *bad = 1;
      B[c.i + j * L] = v;
    }
}

// Solve A X = B (L x L, nrhs columns) by LU; A and B are overwritten (B <- X).
// full=false: partial (row) pivoting on the largest |a| in the column (first
// max); full=true: complete pivoting on the largest |a| of the trailing block,
// first max in column-major order.  Returns false on a zero / non-finite pivot.
template <typename R>
__device__ bool sm_lu_solve(typename SmallMat<R>::M* A, typename SmallMat<R>::M* B, int L, int nrhs, bool full,
                            int* colperm /*smem[L]*/, int* piv /*smem[L]*/) {
  __shared__ int bad;
  __shared__ typename SmallMat<R>::M dinv[kMaxL];
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  if (L <= kWarpL) {
    if (threadIdx.x < 32) lu_solve_team<R, true>(WarpTeam{(int)threadIdx.x, 32}, A, B, L, nrhs, full, piv, dinv, colperm, &bad);
  } else {
    lu_solve_team<R, !std::is_same<R, double>::value>(CtaTeam{(int)threadIdx.x, (int)blockDim.x}, A, B, L, nrhs, full, piv,
                                                      dinv, colperm, &bad);
  }
  __syncthreads();
  const bool ok = !bad;
  __syncthreads();
  return ok;
}

// Cholesky factor and inverse factor in one sweep on a team: H = L D L^H with L
// unit lower triangular, so R = D^1/2 L^H and R^-1 = (L^-1)^H D^-1/2.  One array
// holds both: U = D L^H above (and on) the diagonal, W = L^-1 below it; step k
// takes L_ik U_k out of the rows i > k of U and L_ik W_k out of W's.  A step is a
// reciprocal, a multiplier and an update (no square root in the chain; FP64 on a
// whole CTA takes the multipliers once, see lu_solve_team), and there is no
// second sweep for the inverse.
template <typename R, bool RED, class Team>
__device__ void ldl_team(const Team tm, typename SmallMat<R>::M* U, int L, R* dinv, int* bad) {
  using M = typename SmallMat<R>::M;
  const Cells c(tm.rank, tm.size, L);
  tm.sync();
  for (int k = 0; k < L; ++k) {
    R di;
    const R d = U[k + k * L].x;
    if (!r_pos_finite(d)) { if (tm.rank == 0) *bad = 1; return; }
    if constexpr (RED) {
      di = r_recip(d);
    } else {
      if (tm.rank < 32) {
        di = r_recip(d);
        if (tm.rank == 0) dinv[k] = di;
      }
      tm.sync();
      di = dinv[k];
    }
    if (c.i > k && c.i < L) {
      const M u = U[k + c.i * L];
      const M l = r_recip_ok(d) ? cmake(u.x * di, -(u.y * di)) : m_over(u, d);  // L_ik
      for (int j = c.j0; j < L; j += c.step) {
        if (j > k && j < c.i) continue;  // neither triangle has (i, j) at this step
        M* col = U + j * L;
        col[c.i] = j == k ? m_neg(l) : csub(col[c.i], cmul(l, col[k]));
      }
    }
    tm.sync();
  }
}

// H = R^H R with R upper triangular, real positive diagonal, and Ri = R^-1.
// Rm, Ri and H are three arrays; H (its upper triangle is read) is overwritten.
template <typename R>
__device__ bool sm_chol_inv(typename SmallMat<R>::M* Rm, typename SmallMat<R>::M* Ri, typename SmallMat<R>::M* H, int L) {
  using M = typename SmallMat<R>::M;
  __shared__ int bad;
  __shared__ R dinv[kMaxL];
  if (threadIdx.x == 0) bad = 0;
  const Cells c((int)threadIdx.x, (int)blockDim.x, L);
  if (c.i < L)
    for (int j = c.j0; j < c.i; j += c.step) H[c.i + j * L] = czero<M>();
  __syncthreads();
  if (L <= kWarpL) {
    if (threadIdx.x < 32) ldl_team<R, true>(WarpTeam{(int)threadIdx.x, 32}, H, L, dinv, &bad);
  } else {
    ldl_team<R, !std::is_same<R, double>::value>(CtaTeam{(int)threadIdx.x, (int)blockDim.x}, H, L, dinv, &bad);
  }
  __syncthreads();
  if (bad) return false;  // shared: the same for every thread
  for (int i = threadIdx.x; i < L; i += blockDim.x) dinv[i] = r_recip(r_sqrt(H[i + i * L].x));
  __syncthreads();
  if (c.i < L) {
    const R q = dinv[c.i];
    for (int j = c.j0; j < L; j += c.step) {
      const M v = H[c.i + j * L];
      const M w = cmake(v.x * q, v.y * q);
      if (j >= c.i) {  // R_ij = U_ij / sqrt(d_i); and zero below the diagonal of R and Ri
        Rm[c.i + j * L] = j == c.i ? cmake(r_sqrt(v.x), r_const<R>(0.0f)) : w;
        if (j == c.i) Ri[c.i + j * L] = cmake(q, r_const<R>(0.0f));
        else { Rm[j + c.i * L] = czero<M>(); Ri[j + c.i * L] = czero<M>(); }
      } else {
        Ri[j + c.i * L] = cmake(w.x, -w.y);  // R^-1_ji = conj(W_ij) / sqrt(d_i)
      }
    }
  }
  __syncthreads();
  return true;
}

// Frobenius norm in FP64 (any scale): per-thread sums of |m|^2, a warp
// shuffle tree, then the warps' sums in order (deterministic).
template <typename R> __device__ double sm_fro(const typename SmallMat<R>::M* Mm, int LL) {
  __shared__ double wsum[kSmallThreads / 32];
  __shared__ double r;
  double s = 0.0;
  for (int e = threadIdx.x; e < LL; e += blockDim.x) s += cabs2(m_to_double2(Mm[e]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = wsum[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) t += wsum[w];
    r = sqrt(t);
  }
  __syncthreads();
  const double v = r;
  __syncthreads();
  return v;
}

}  // namespace bdda
