// 64-bit fixed-point FFT core of the FP64 and double-float block MVPs and of
// the Green spectrum.
//
// GB300 runs FP64 at 1/64 of its FP32 rate (2 operations per clock and SM),
// but 64-bit integer additions at about 31 and 32 x 32 -> 64-bit
// multiply-adds at 24-32.  An FFT needs no floating point between its input
// and its output: a line is converted once to 64-bit fixed point with one
// power-of-two scale for the whole line, transformed with integer additions
// and 62-bit twiddle products, and converted back.  Measured (arithmetic
// alone, per clock and SM): complex product 0.46 FP64 -> 2.1, addition 1.7 ->
// 31.  The scale leaves the largest value 2-7 bits more than FP64's 53, so the
// rounding errors stay below those of the FP64 transform
// (tests/test_fixed_point_fft.py measures both against extended precision).
//
// Values are integers v with a common exponent: |z| <= 2^62 for every complex
// value of a line at any point of its transform, sums inside a butterfly
// included (a product's three partial sums then stay below 2^63).  Twiddles and spectra are Q62 integers split as
// h 2^32 + l with signed l, so a product is three 32 x 32 -> 64 multiplies
// (l l would reach one unit of the last place and is dropped).  The twiddle
// product of a radix-R stage also divides by 2^floor(log2 R), which undoes most
// of the butterfly's worst-case growth at no cost: the shift that a Q62
// product needs anyway becomes shorter.
//
// The transform pair is fft_core.cuh's: forward decimation in frequency
// (natural in, digit-reversed out), inverse its adjoint in reverse order.  One
// warp transforms NL lines in shared memory in place.
#pragma once

#include "common.cuh"

#if defined(__CUDACC__)
#define BDDA_FX_FN __device__ __forceinline__
#define BDDA_FX_SYNCWARP() __syncwarp()
#else
#define BDDA_FX_FN inline
#define BDDA_FX_SYNCWARP() ((void)0)
#endif

namespace bdda {
namespace fx {

// Complex fixed-point value (the size of a complex FP64 value, whose bits the
// same shared-memory slots hold before and after the transform).
struct __align__(16) Val { long long x, y; };
// Complex Q62 factor, each part h 2^32 + l with l signed.
struct __align__(16) Fac { int rh, rl, ih, il; };

constexpr int kTopBit = 62;  // |z| <= 2^kTopBit

BDDA_FX_FN Fac ldfac(const Fac* p) {
#if defined(__CUDA_ARCH__)
  const int4 v = __ldg(reinterpret_cast<const int4*>(p));
  return {v.x, v.y, v.z, v.w};
#else
  return *p;
#endif
}
BDDA_FX_FN Val add(Val a, Val b) { return {a.x + b.x, a.y + b.y}; }
BDDA_FX_FN Val sub(Val a, Val b) { return {a.x - b.x, a.y - b.y}; }
// 32 x 32 -> 64-bit product as one instruction: from plain C++ the compiler
// widens the factors and multiplies 64 x 64 (36 instead of 12 multiplies per
// complex product, 0.95 -> 0.49 clocks).  Products are added with 64-bit adds:
// the multiply-add form takes 2.75 slots of the multiplier pipe, which bounds
// these kernels, instead of 2.
BDDA_FX_FN long long mw(int a, int b) {
#if defined(__CUDA_ARCH__)
  long long d;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
  return d;
#else
  return (long long)a * b;
#endif
}
BDDA_FX_FN long long shl(long long v, int s) { return (long long)((unsigned long long)v << s); }
BDDA_FX_FN void split(long long v, int& h, int& l) {
  l = (int)v;
  h = (int)(v >> 32) + (int)((unsigned)v >> 31);
}
// v / 2^s rounded, s >= 1
BDDA_FX_FN long long shr_round(long long v, int s) { return (v + (1ll << (s - 1))) >> s; }

constexpr int hi_of(long long q) { return (int)((q + 0x80000000ll) >> 32); }
constexpr int lo_of(long long q) { return (int)q; }

// v times the real constant Q / 2^62
template <long long Q> BDDA_FX_FN long long mulk(long long v) {
  int h, l;
  split(v, h, l);
  const long long c = mw(h, lo_of(Q)) + mw(l, hi_of(Q)) + (1ll << 29);
  return shl(mw(h, hi_of(Q)), 2) + (c >> 30);
}

// z times the complex factor (rh, rl) + i (ih, il), conjugated with CJ, over 2^D
template <int D, bool CJ> BDDA_FX_FN Val cmul(Val z, int rh, int rl, int ih, int il) {
  int xh, xl, yh, yl;
  split(z.x, xh, xl);
  split(z.y, yh, yl);
  const long long rnd = D >= 2 ? (1ll << 31) : (1ll << (29 + D));
  // real: x r -+ y i; imaginary: y r +- x i
  const long long a = mw(xh, rl) + mw(xl, rh) + rnd, b = mw(yh, il) + mw(yl, ih);
  const long long c = mw(yh, rl) + mw(yl, rh) + rnd, d = mw(xh, il) + mw(xl, ih);
  const long long e = mw(xh, rh), f = mw(yh, ih), g = mw(yh, rh), k = mw(xh, ih);
  const long long cr = CJ ? a + b : a - b, ci = CJ ? c - d : c + d;
  const long long mr = CJ ? e + f : e - f, mi = CJ ? g - k : g + k;
  if constexpr (D < 2) return {shl(mr, 2 - D) + (cr >> (30 + D)), shl(mi, 2 - D) + (ci >> (30 + D))};
  else if constexpr (D == 2) return {mr + (cr >> 32), mi + (ci >> 32)};
  else return {(mr + (cr >> 32) + (1ll << (D - 3))) >> (D - 2), (mi + (ci >> 32) + (1ll << (D - 3))) >> (D - 2)};
}

// Sum of complex products Fac x Val, scaled as its Val operands; one shift and rounding at the end.
struct Split { int xh, xl, yh, yl; };
BDDA_FX_FN Split split(Val v) {
  Split s;
  split(v.x, s.xh, s.xl);
  split(v.y, s.yh, s.yl);
  return s;
}
struct Acc {
  long long cr = 1ll << 29, ci = 1ll << 29, mr = 0, mi = 0;
  BDDA_FX_FN void mad(const Fac& g, const Split& s) {
    cr += (mw(s.xh, g.rl) + mw(s.xl, g.rh)) - (mw(s.yh, g.il) + mw(s.yl, g.ih));
    mr += mw(s.xh, g.rh) - mw(s.yh, g.ih);
    ci += (mw(s.xh, g.il) + mw(s.xl, g.ih)) + (mw(s.yh, g.rl) + mw(s.yl, g.rh));
    mi += mw(s.xh, g.ih) + mw(s.yh, g.rh);
  }
  // the products are subtracted: a low half of -2^31 has no negative in 32 bits
  BDDA_FX_FN void msub(const Fac& g, const Split& s) {
    cr -= (mw(s.xh, g.rl) + mw(s.xl, g.rh)) - (mw(s.yh, g.il) + mw(s.yl, g.ih));
    mr -= mw(s.xh, g.rh) - mw(s.yh, g.ih);
    ci -= (mw(s.xh, g.il) + mw(s.xl, g.ih)) + (mw(s.yh, g.rl) + mw(s.yl, g.rh));
    mi -= mw(s.xh, g.ih) + mw(s.yh, g.rh);
  }
  BDDA_FX_FN Val get() const { return {shl(mr, 2) + (cr >> 30), shl(mi, 2) + (ci >> 30)}; }
  // this sum plus or minus another one (of no rounding half), whose middle sums together may pass 2^63
  BDDA_FX_FN Val get(const Acc& o, bool sub) const {
    const long long hr = o.cr >> 1, hi = o.ci >> 1;
    return {shl(sub ? mr - o.mr : mr + o.mr, 2) + (((cr >> 1) + (sub ? -hr : hr)) >> 29),
            shl(sub ? mi - o.mi : mi + o.mi, 2) + (((ci >> 1) + (sub ? -hi : hi)) >> 29)};
  }
};

// Index of the spectrum components that couple component c to row r, r and c < 3: of the symmetric block A (xx xy xz yy yz
// zz), and with f = 6, [A B; -B A], of the antisymmetric B (xy xz yz, -1 on its diagonal; subtracted where r > c).
BDDA_FX_FN constexpr int green_a(int r, int c) { return r + c + (r != 0 && c != 0 ? 1 : 0); }
BDDA_FX_FN constexpr int green_b(int r, int c) { return r == c ? -1 : 5 + r + c; }
// Bits that a spectrum component stays below 1, and that values are shifted for the products at least: the middle sums of
// three terms stay below 7.3 2^60, of f = 6's other two below 4.9, and a row of five below 5 2^60, which the shift to the
// inverse transform's headroom takes.  Each bit costs precision, the first against elements far below a line's peak: with
// 3 and 2 bits f = 6 had errors of 2.8e-16 (N=568, extended precision), with 2 and 2 1.7e-16.
constexpr int kGreenBits = 1, kProductBits = 1;

// ---- butterflies: forward exp(-2 pi i / R), INV exp(+2 pi i / R) --------------
constexpr long long kS60 = 3993837246235628775ll;   // sin 60, Q62
constexpr long long kHalfRt = 3260954456333195553ll;  // sqrt(1/2)
constexpr long long kRt5_4 = 2578010857022246787ll;   // sqrt(5) / 4
constexpr long long kS72 = 4385974038932618941ll, kS36 = 2710681029835013083ll;
constexpr long long kC9[3] = {3532756447825785444ll, 800810873071977681ll, -4333567320897763126ll};  // cos 40 k, k = 1, 2, 4
constexpr long long kS9[3] = {2964334632409774423ll, 4541624145405292212ll, 1577289512995517789ll};

BDDA_FX_FN Val mul_i(Val a) { return {-a.y, a.x}; }
BDDA_FX_FN Val mul_mi(Val a) { return {a.y, -a.x}; }
// a -+ i b forward / inverse as the pair (a - i b, a + i b) or its swap
template <bool INV> BDDA_FX_FN void pm_i(Val a, Val b, Val& minus, Val& plus) {
  const Val p = {a.x + b.y, a.y - b.x}, m = {a.x - b.y, a.y + b.x};  // a - i b, a + i b
  minus = INV ? m : p;
  plus = INV ? p : m;
}

template <bool INV> BDDA_FX_FN void dft2(Val* v) {
  const Val a = v[0], b = v[1];
  v[0] = add(a, b);
  v[1] = sub(a, b);
}
template <bool INV> BDDA_FX_FN void dft3(Val* v) {
  const Val t = add(v[1], v[2]), d = sub(v[1], v[2]);
  const Val h = {v[0].x - (t.x >> 1), v[0].y - (t.y >> 1)};
  const Val s = {mulk<kS60>(d.x), mulk<kS60>(d.y)};
  v[0] = add(v[0], t);
  pm_i<INV>(h, s, v[1], v[2]);
}
template <bool INV> BDDA_FX_FN void dft4(Val* v) {
  const Val a0 = add(v[0], v[2]), a1 = sub(v[0], v[2]);
  const Val b0 = add(v[1], v[3]), b1 = sub(v[1], v[3]);
  v[0] = add(a0, b0);
  v[2] = sub(a0, b0);
  pm_i<INV>(a1, b1, v[1], v[3]);
}
// s a + t b and t a - s b for the constants s = sin 72, t = sin 36 (one split per value)
BDDA_FX_FN void rot5(long long a, long long b, long long& p, long long& q) {
  int ah, al, bh, bl;
  split(a, ah, al);
  split(b, bh, bl);
  constexpr int sh = hi_of(kS72), sl = lo_of(kS72), th = hi_of(kS36), tl = lo_of(kS36);
  const long long c = mw(ah, sl) + mw(al, sh) + (mw(bh, tl) + mw(bl, th)) + (1ll << 29);
  const long long d = mw(ah, tl) + mw(al, th) + (mw(bh, -sl) + mw(bl, -sh)) + (1ll << 29);
  p = shl(mw(ah, sh) + mw(bh, th), 2) + (c >> 30);
  q = shl(mw(ah, th) + mw(bh, -sh), 2) + (d >> 30);
}
template <bool INV> BDDA_FX_FN void dft5(Val* v) {
  const Val t1 = add(v[1], v[4]), t2 = add(v[2], v[3]), t3 = sub(v[1], v[4]), t4 = sub(v[2], v[3]);
  const Val t = add(t1, t2), u = sub(t1, t2);
  // cos 72 and cos 144 are -1/4 +- sqrt(5)/4
  const Val a = {v[0].x - (t.x >> 2), v[0].y - (t.y >> 2)};
  const Val e = {mulk<kRt5_4>(u.x), mulk<kRt5_4>(u.y)};
  Val b1, b2;
  rot5(t3.x, t4.x, b1.x, b2.x);
  rot5(t3.y, t4.y, b1.y, b2.y);
  v[0] = add(v[0], t);
  pm_i<INV>(add(a, e), b1, v[1], v[4]);
  pm_i<INV>(sub(a, e), b2, v[2], v[3]);
}
// z exp(-+ i pi / 4)
template <bool INV> BDDA_FX_FN Val rot8(Val z) {
  return INV ? Val{mulk<kHalfRt>(z.x - z.y), mulk<kHalfRt>(z.x + z.y)}
             : Val{mulk<kHalfRt>(z.x + z.y), mulk<kHalfRt>(z.y - z.x)};
}
template <bool INV> BDDA_FX_FN void dft8(Val* v) {
  Val a[4], b[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    a[r] = add(v[r], v[r + 4]);
    b[r] = sub(v[r], v[r + 4]);
  }
  b[1] = rot8<INV>(b[1]);
  b[2] = INV ? mul_i(b[2]) : mul_mi(b[2]);
  b[3] = rot8<INV>(INV ? mul_i(b[3]) : mul_mi(b[3]));
  dft4<INV>(a);
  dft4<INV>(b);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    v[2 * m] = a[m];
    v[2 * m + 1] = b[m];
  }
}
template <bool INV, long long QC, long long QS> BDDA_FX_FN Val rotk(Val z) {
  // forward exp(-i a), inverse exp(+i a), a the angle with cosine QC and sine QS
  return cmul<0, !INV>(z, hi_of(QC), lo_of(QC), hi_of(QS), lo_of(QS));
}
// 9 = 3 x 3 with constant twiddles
template <bool INV> BDDA_FX_FN void dft9(Val* v) {
  Val y[3][3];
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    Val u[3] = {v[n], v[n + 3], v[n + 6]};
    dft3<INV>(u);
    y[n][0] = u[0]; y[n][1] = u[1]; y[n][2] = u[2];
  }
  y[1][1] = rotk<INV, kC9[0], kS9[0]>(y[1][1]);
  y[1][2] = rotk<INV, kC9[1], kS9[1]>(y[1][2]);
  y[2][1] = rotk<INV, kC9[1], kS9[1]>(y[2][1]);
  y[2][2] = rotk<INV, kC9[2], kS9[2]>(y[2][2]);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    Val u[3] = {y[0][k], y[1][k], y[2][k]};
    dft3<INV>(u);
    v[k] = u[0]; v[k + 3] = u[1]; v[k + 6] = u[2];
  }
}

template <int R, bool INV> BDDA_FX_FN void dft(Val* v);
constexpr int inv_mod(int a, int m) {
  for (int x = 1; x < m; ++x)
    if (a * x % m == 1) return x;
  return 1;
}
// R = A B with coprime factors: index maps instead of twiddles (Good 1958):
// input B n1 + A n2, output k with k = k1 mod A, k = k2 mod B.
template <int A, int B, bool INV> BDDA_FX_FN void dft_pfa(Val* v) {
  constexpr int R = A * B;
  Val y[A][B];
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
    Val u[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) u[n1] = v[(B * n1 + A * n2) % R];
    dft<A, INV>(u);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) y[k1][n2] = u[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    Val u[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) u[n2] = y[k1][n2];
    dft<B, INV>(u);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) v[(k1 * B * inv_mod(B % A, A) + k2 * A * inv_mod(A % B, B)) % R] = u[k2];
  }
}
template <int R, bool INV> BDDA_FX_FN void dft(Val* v) {
  if constexpr (R == 2) dft2<INV>(v);
  else if constexpr (R == 3) dft3<INV>(v);
  else if constexpr (R == 4) dft4<INV>(v);
  else if constexpr (R == 5) dft5<INV>(v);
  else if constexpr (R == 6) dft_pfa<2, 3, INV>(v);
  else if constexpr (R == 8) dft8<INV>(v);
  else if constexpr (R == 9) dft9<INV>(v);
  else {
    static_assert(R == 10, "register radix");
    dft_pfa<2, 5, INV>(v);
  }
}

// ---- plan ----------------------------------------------------------------------
constexpr int kMaxFxStages = 8;
constexpr BDDA_HD int flog2(int r) { return r >= 8 ? 3 : r >= 4 ? 2 : 1; }

BDDA_HD int div_magic(int q, int m) { return (int)((unsigned)(q * m) >> 21); }

// Radix schedule and shared-memory layout of one axis: element idx lives at
// (idx / Rl) S + idx % Rl, S odd, so that the lanes of the last stage (S apart)
// and of the others (adjacent) touch the eight 16-byte bank groups evenly;
// lines are LW (odd) apart for the transposed tile copies.
struct Plan {
  int N, nst, Rl, S, LW;
  int radix[kMaxFxStages], M[kMaxFxStages], two[kMaxFxStages];  // two: offset of the stage's twiddles
  // q / d as (q m) >> 21 with m = ceil(2^21 / d), exact for q < 1800, d <= 600 (no float conversions, which run
  // at a quarter of the integer rate): d = M[s], the butterflies N / radix[s] of a line, Rl
  int mM[kMaxFxStages], mB[kMaxFxStages], mRl;
  int D;          // bits divided away by the twiddle products of a whole transform
  // headroom bits of the largest input value, forward and inverse: growth by the end, and before the last butterfly
  int head[2], early[2];
  BDDA_FX_FN int addr(int i) const {
    const int q = div_magic(i, mRl);
    return q * S + (i - q * Rl);
  }
  // Headroom of a line whose values sum to at most 2^c times the bound of a single one: no sum of them grows past 2^c,
  // nor past 2^(c - D) after the divisions.
  BDDA_FX_FN int headroom(bool inv, int c) const {
    const int h = c - D > early[inv] ? c - D : early[inv];
    const int m = h < head[inv] ? h : head[inv];
    return m < c ? m : c;
  }
};

// ---- FP64 <-> fixed -------------------------------------------------------------
BDDA_FX_FN int clz32(int a) {
#if defined(__CUDA_ARCH__)
  return __clz(a);
#else
  return a ? __builtin_clz((unsigned)a) : 32;
#endif
}
// Magnitude key of a complex FP64 value's parts (bits): compares like |v|, 0 only for zero.
BDDA_FX_FN int key(long long bits) { return (int)((bits >> 32) & 0x7fffffff) | ((int)bits != 0 ? 1 : 0); }

// A part's size in units of 2^-19 of the line's largest power of two, rounded up (E: exponent field of the largest key).
// Their sum over a line bounds every value of its transform: headroom sum_head(sum) bits.
BDDA_FX_FN int sum_unit(long long bits, int E) {
  const int k = (int)((bits >> 32) & 0x7fffffff), e = k >> 20;
  const int r = E - e + 1;
  return ((k & 0xfffff) | (e ? 0x100000 : 0)) >> (r > 31 ? 31 : r < 1 ? 1 : r);
}
BDDA_FX_FN int sum_head(unsigned sum, int count) {  // count: values summed, two rounded-up parts each
  sum += 2 * (unsigned)count;
  const int b = sum <= 1 ? 0 : 32 - clz32((int)(sum - 1));  // sum <= 2^b
  return b > 21 ? b - 21 : 0;
}
// Lines whose largest value is below 2^-923 (subnormals among them) are scaled up by 2^200 first.
constexpr int kTinyKey = 100 << 20;
BDDA_FX_FN bool tiny(int kmax) { return kmax > 0 && kmax < kTinyKey; }

BDDA_HD double bits_to_double(long long b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double(b);
#else
  double d;
  __builtin_memcpy(&d, &b, 8);
  return d;
#endif
}
BDDA_HD long long double_to_bits(double d) {
#if defined(__CUDA_ARCH__)
  return __double_as_longlong(d);
#else
  long long b;
  __builtin_memcpy(&b, &d, 8);
  return b;
#endif
}
BDDA_FX_FN Val lift_tiny(Val v) {
  return {double_to_bits(bits_to_double(v.x) * 0x1p200), double_to_bits(bits_to_double(v.y) * 0x1p200)};
}

// Scale of a line: largest key, headroom bits below kTopBit.
struct Scale {
  int rsh0;   // right shift of a value with exponent field e: rsh0 - e
  int ebase;  // result exponent: value = fixed * 2^ebase (before the transform's divisions)
  bool zero, bad;
};
BDDA_FX_FN Scale make_scale(int kmax, int head) {
  Scale s;
  s.zero = kmax == 0;
  s.bad = kmax >= 0x7ff00000;  // infinity or NaN in the line
  const int E = (kmax >> 20) > 1 ? (kmax >> 20) : 1;
  const int sh = kTopBit - 54 - head;  // |z| < sqrt(2) 2^53 2^sh
  s.rsh0 = 10 - sh + E;
  s.ebase = E - 1075 - sh;
  return s;
}
BDDA_FX_FN long long from_bits(long long b, int rsh0) {
  const int hi = (int)(b >> 32), e0 = (hi >> 20) & 0x7ff;
  const int e = e0 ? e0 : 1;
  const unsigned long long m = ((unsigned long long)((hi & 0xfffff) | (e0 ? 0x100000 : 0)) << 32 | (unsigned)b) << 10;
  const int r = rsh0 - e;  // >= 1
  const long long a = (long long)(((m >> (r > 63 ? 63 : r - 1)) + 1) >> 1);
  return b < 0 ? -a : a;
}
BDDA_FX_FN int clz64(unsigned long long a) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)a);
#else
  return a ? __builtin_clzll(a) : 64;
#endif
}
// v 2^eb rounded to FP64 (bits)
BDDA_FX_FN long long to_bits(long long v, int eb) {
  if (v == 0) return 0;
  const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int lz = clz64(a);
  const unsigned long long m = a << lz;
  const unsigned long long r = (m >> 11) + ((m >> 10) & 1);  // 53 bits with the leading one, or 2^53
  const int be = 1086 - lz + eb;                             // exponent field
  if (be < 1 || be > 2046) {                                 // below the normal range, or above it
    const double d = ldexp((double)(long long)r, be - 1075);
    return double_to_bits(v < 0 ? -d : d);
  }
  return (long long)(((unsigned long long)(be - 1) << 52) + r) | (v & (long long)0x8000000000000000ull);
}
constexpr long long kNaNBits = 0x7ff8000000000000ll;

// What the output of a line's transform needs: its exponent, or that it is all zero or not finite.
BDDA_FX_FN Val to_bits(Val v, int eb, bool bad) {
  if (bad) return {kNaNBits, kNaNBits};
  return {to_bits(v.x, eb), to_bits(v.y, eb)};
}

// ---- block-scaled lines ------------------------------------------------------------
// Between the passes a line is kept in fixed point with an exponent of its
// own: parts below 2^kStoreBit, the largest in [2^(kStoreBit - 1), 2^kStoreBit)
// (or, below 2^32, shifted up as far as that takes it), value = v 2^e.
constexpr int kStoreBit = 62;
// Both marks are exponents like any other to the shifts of an element against its line's largest, which stay in range.
constexpr int kBadExp = 1 << 24;          // a line that is not finite
constexpr int kZeroExp = -(1 << 20);      // a line of zeros
// OR of the folded high words of values: the bits in use.
BDDA_FX_FN int bits_of(Val v) {
  const int a = (int)(v.x >> 32), b = (int)(v.y >> 32);
  return (a ^ (a >> 31)) | (b ^ (b >> 31));
}
// Left shift that brings a line with the given bits in use to kStoreBit.
BDDA_FX_FN int store_shift(int used) { return clz32(used) - (64 - kStoreBit); }
// Right shift, at least 1, that brings values with the given bits in use to a transform's headroom (parts below
// 2^(kTopBit - 1 - head)).
BDDA_FX_FN int fit_shift(int used, int head) {
  const int s = 64 - clz32(used) - (kTopBit - 1 - head);
  return s > 1 ? s : 1;
}
// v / 2^r rounded, r >= 1.
BDDA_FX_FN Val align(Val v, int r) {
  r = r > 62 ? 62 : r;  // (2^62 + 2^61) >> 62 = 1 at most
  const long long half = 1ll << (r - 1);
  return {(v.x + half) >> r, (v.y + half) >> r};
}

// ---- stages ---------------------------------------------------------------------
// Input of a stage: RAW: FP64 bits to convert with the line's scale (rsh[j]),
// FIXED, SHIFT: fixed values to shift right by rsh[j] (left where negative),
// ALIGN: stored values of element exponents ex[j * exs + idx], shifted right by rsh[j] - ex.
enum In { kRaw, kFixed, kShift, kAlign };
struct InArgs {
  const int* rsh;
  const int* ex;
  int exs;
};

// One stage over NL lines of a warp (line j at s + j p.LW).  PRUNE: only
// elements idx < nv (nv <= N / 2) are read (forward) or written (inverse), so
// butterfly elements i with 2 i >= R are compile-time zeros or dead.  used
// (USED: the last stage): line j's bits in use at used[j].
template <int R, bool INV, int NL, int IN, bool PRUNE, bool USED>
BDDA_FX_FN void stage(Val* __restrict__ s, const Plan& p, int st, const Fac* __restrict__ tw, int lane, int lanes, int nv,
                      const InArgs& in, int* used) {
  constexpr int D = flog2(R);
  const int M = p.M[st], nb = p.N / R, mM = p.mM[st], mB = p.mB[st];
  const int off = st == p.nst - 1 ? 1 : (M / p.Rl) * p.S;
  const Fac* tws = tw + p.two[st];
  for (int t = lane; t < NL * nb; t += lanes) {
    const int j = NL == 1 ? 0 : div_magic(t, mB);
    const int u = t - j * nb;
    const int b = div_magic(u, mM);
    const int n1 = u - b * M, idx0 = b * M * R + n1;
    Val* q = s + j * p.LW + p.addr(idx0);
    Val v[R];
    const int rs = IN == kFixed ? 0 : NL == 3 && j == 2 ? in.rsh[NL - 1] : NL > 1 && j ? in.rsh[NL > 1] : in.rsh[0];  // rsh[j]
    const int* ex = IN == kAlign ? in.ex + j * in.exs + idx0 : nullptr;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (PRUNE && !INV && (2 * i >= R || idx0 + i * M >= nv)) {
        v[i] = Val{0, 0};
        continue;
      }
      v[i] = q[i * off];
      if (IN == kRaw) v[i] = Val{from_bits(v[i].x, rs), from_bits(v[i].y, rs)};
      if (IN == kShift) v[i] = rs > 0 ? Val{shr_round(v[i].x, rs), shr_round(v[i].y, rs)} : Val{shl(v[i].x, -rs), shl(v[i].y, -rs)};
      if (IN == kAlign) v[i] = align(v[i], rs - ex[i * M]);
    }
    const bool twid = M > 1;
    if (INV && twid) {
      v[0] = Val{shr_round(v[0].x, D), shr_round(v[0].y, D)};
#pragma unroll
      for (int k = 1; k < R; ++k) {
        const Fac w = ldfac(tws + (k - 1) * M + n1);
        v[k] = cmul<D, true>(v[k], w.rh, w.rl, w.ih, w.il);
      }
    }
    dft<R, INV>(v);
    if (!INV && twid) {
      v[0] = Val{shr_round(v[0].x, D), shr_round(v[0].y, D)};
#pragma unroll
      for (int k = 1; k < R; ++k) {
        const Fac w = ldfac(tws + (k - 1) * M + n1);
        v[k] = cmul<D, false>(v[k], w.rh, w.rl, w.ih, w.il);
      }
    }
    int o = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (PRUNE && INV && (2 * i >= R || idx0 + i * M >= nv)) continue;
      q[i * off] = v[i];
      if (USED) o |= bits_of(v[i]);
    }
    if (USED) {
#pragma unroll
      for (int k = 0; k < NL; ++k) used[k] |= j == k ? o : 0;
    }
  }
  BDDA_FX_SYNCWARP();
}

template <bool INV, int NL, int IN, bool PRUNE, bool USED>
BDDA_FX_FN void stage_any(Val* s, const Plan& p, int st, const Fac* tw, int lane, int lanes, int nv, const InArgs& in, int* used) {
  switch (p.radix[st]) {
    case 2: stage<2, INV, NL, IN, PRUNE, USED>(s, p, st, tw, lane, lanes, nv, in, used); break;
    case 3: stage<3, INV, NL, IN, PRUNE, USED>(s, p, st, tw, lane, lanes, nv, in, used); break;
    case 4: stage<4, INV, NL, IN, PRUNE, USED>(s, p, st, tw, lane, lanes, nv, in, used); break;
    case 5: stage<5, INV, NL, IN, PRUNE, USED>(s, p, st, tw, lane, lanes, nv, in, used); break;
    case 6: stage<6, INV, NL, IN, PRUNE, USED>(s, p, st, tw, lane, lanes, nv, in, used); break;
    case 8: stage<8, INV, NL, IN, PRUNE, USED>(s, p, st, tw, lane, lanes, nv, in, used); break;
    case 9: stage<9, INV, NL, IN, PRUNE, USED>(s, p, st, tw, lane, lanes, nv, in, used); break;
    default: stage<10, INV, NL, IN, PRUNE, USED>(s, p, st, tw, lane, lanes, nv, in, used); break;
  }
}

// Forward transform of NL lines, input as IN says, fixed point out, the bits
// in use of its output where USED.  PRUNE: only the first nv <= N / 2 inputs
// are read, the rest are zero.
template <int NL, int IN, bool PRUNE, bool USED>
BDDA_FX_FN void forward(Val* s, const Plan& p, const Fac* tw, int lane, int lanes, int nv, const InArgs& in, int* used) {
  if (p.nst == 1) {
    stage_any<false, NL, IN, PRUNE, USED>(s, p, 0, tw, lane, lanes, nv, in, used);
    return;
  }
  stage_any<false, NL, IN, PRUNE, false>(s, p, 0, tw, lane, lanes, nv, in, used);
  for (int st = 1; st < p.nst - 1; ++st) stage_any<false, NL, kFixed, false, false>(s, p, st, tw, lane, lanes, nv, in, used);
  stage_any<false, NL, kFixed, false, USED>(s, p, p.nst - 1, tw, lane, lanes, nv, in, used);
}
// Inverse transform, only the first nv <= N / 2 outputs written.
template <int NL, int IN, bool USED>
BDDA_FX_FN void inverse(Val* s, const Plan& p, const Fac* tw, int lane, int lanes, int nv, const InArgs& in, int* used) {
  if (p.nst == 1) {
    stage_any<true, NL, IN, true, USED>(s, p, 0, tw, lane, lanes, nv, in, used);
    return;
  }
  stage_any<true, NL, IN, false, false>(s, p, p.nst - 1, tw, lane, lanes, nv, in, used);
  for (int st = p.nst - 2; st >= 1; --st) stage_any<true, NL, kFixed, false, false>(s, p, st, tw, lane, lanes, nv, in, used);
  stage_any<true, NL, kFixed, true, USED>(s, p, 0, tw, lane, lanes, nv, in, used);
}

}  // namespace fx
}  // namespace bdda
