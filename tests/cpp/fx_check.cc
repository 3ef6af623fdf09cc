// Host check of the fixed-point kernel value (csrc/ds_fx.cuh): the largest
// relative error of exp(-arg) over arguments in [0, 48), and of whole pair
// values against long double, printed as "exp_err pair_err".
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "fx_tables.h"

static double from_bits(uint64_t b) {
  double d;
  std::memcpy(&d, &b, sizeof(d));
  return d;
}

static uint64_t s = 88172645463325252ull;
static uint64_t rnd() {
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s;
}
static double uni(double a, double b) { return a + (b - a) * (double)(rnd() >> 11) * 0x1p-53; }

int main() {
  const std::vector<uint64_t> t = ds::fx_tables();
  const uint64_t *t1 = t.data(), *t2 = t.data() + ds::FX_T1;
  if (from_bits(ds::fx_exp_bits(0, t1, t2)) != 1.0) return 1;
  long double worst = 0;
  auto one = [&](uint64_t arg) {
    const long double want = expl(-ldexpl((long double)arg, -56));
    const long double e = fabsl((long double)from_bits(ds::fx_exp_bits(arg, t1, t2)) / want - 1);
    if (e > worst) worst = e;
  };
  for (int k = 0; k < 2000000; ++k) one((uint64_t)(uni(0, 48) * 0x1p56));
  for (int j = 0; j < 48 * 32; ++j)  // around every table step
    for (int64_t d = -3; d <= 3; ++d)
      if (j > 0 || d >= 0) one(((uint64_t)j << 51) + (uint64_t)d);
  for (int k = 0; k < 60; ++k) one(1ull << (k < 56 ? k : 55));
  // whole values: coordinates up to `big`, separations of a few units
  long double pair = 0;
  auto fma_ = [](double a, double b, double c) { return std::fma(a, b, c); };
  auto ll = [](double v) { return (int64_t)llrint(v); };
  for (double big : {1.0, 600.0, 1e5}) {
    const double c[3] = {0.08, 0.08, 0.125}, o = big / 3;
    for (int k = 0; k < 200000; ++k) {
      long double arg = 0;
      uint64_t d[3];
      for (int a = 0; a < 3; ++a) {
        const double sh = std::sqrt(c[a]), sl = std::fma(-sh, sh, c[a]) / (2 * sh);
        const double x = uni(0, big), y = x + uni(-8, 8);
        auto fix = [&](double v) {
          const double w = v - o, bb = w - v, err = (v - (w - bb)) + (-o - bb);
          return ds::fx_coord(w, err, sh, sl, fma_, ll);
        };
        d[a] = fix(x) - fix(y);
        const long double dd = (long double)x - (long double)y;
        arg += (long double)c[a] * dd * dd;
      }
      if (arg >= 47.9L) continue;
      const uint64_t g = ds::fx_exp_bits(ds::fx_arg(d[0], d[1], d[2]), t1, t2);
      const long double e = fabsl((long double)from_bits(g) / expl(-arg) - 1);
      if (e > pair) pair = e;
    }
  }
  std::printf("%.3Le %.3Le\n", worst, pair);
  return 0;
}
