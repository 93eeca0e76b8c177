// The fixed-point arithmetic of the FP64 and double-float block MVPs, compiled for the host from the device source
// (tests/test_fixed_point_arith.py).
#include <cmath>

#include "fx_fft.cuh"

using namespace bdda;

extern "C" {

// Sum of n products of Q62 factors g (re, im) and values z, those with sub[i] subtracted; from the fourth on in a sum of
// their own that is added at the end (minus: subtracted).
void fx_products(int n, const long long* g, const long long* z, const int* sub, int minus, long long* out) {
  fx::Acc acc, rest{0, 0, 0, 0};
  for (int i = 0; i < n; ++i) {
    fx::Fac f;
    fx::split(g[2 * i], f.rh, f.rl);
    fx::split(g[2 * i + 1], f.ih, f.il);
    const fx::Split s = fx::split(fx::Val{z[2 * i], z[2 * i + 1]});
    fx::Acc& a = i < 3 ? acc : rest;
    if (sub[i]) a.msub(f, s);
    else a.mad(f, s);
  }
  const fx::Val v = n > 3 ? acc.get(rest, minus != 0) : acc.get();
  out[0] = v.x;
  out[1] = v.y;
}

// Exponents that mark a line of zeros and one that is not finite.
int fx_zero_exp() { return fx::kZeroExp; }
int fx_bad_exp() { return fx::kBadExp; }
// v / 2^r, rounded
long long fx_align(long long v, int r) { return fx::align(fx::Val{v, 0}, r).x; }

}  // extern "C"
