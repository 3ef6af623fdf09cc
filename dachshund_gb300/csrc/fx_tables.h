// The fixed-point exponential's tables (ds_fx.cuh), from the host's long double
// exponential (64 bits of mantissa or more).
#pragma once

#include <cmath>
#include <cstdint>
#include <vector>

#include "ds_fx.cuh"

namespace ds {

// T1 then T2.  T1[j]: the mantissa of exp(-j / 32) in [2^62, 2^63) with its
// exponent in the low FX_EXP_BITS bits, the nearest such number; T2[i]: exp(-i /
// 4096) in units of 2^-64 (1 as 2^64 - 1).
inline std::vector<uint64_t> fx_tables() {
  std::vector<uint64_t> t(FX_T1 + FX_T2);
  long double whole[50], part[32];
  for (int i = 0; i < 50; ++i) whole[i] = expl(-(long double)i);
  for (int i = 0; i < 32; ++i) part[i] = expl(-(long double)i / 32);
  const uint64_t step = 1ull << FX_EXP_BITS;
  for (int j = 0; j < FX_T1; ++j) {
    int e;
    // v = f 2^e, f in [0.5, 1): mantissa f 2^63, value mantissa 2^-62 2^(e - 1)
    const long double f = frexpl(whole[j / 32] * part[j % 32], &e);
    const uint64_t ex = (uint64_t)(1 - e);
    const uint64_t m = (uint64_t)rintl((ldexpl(f, 63) - (long double)ex) / (long double)step);
    t[j] = m * step + ex;
  }
  for (int i = 0; i < FX_T2; ++i) {
    const long double v = ldexpl(expl(-(long double)i / 4096), 64);
    t[FX_T1 + i] = i == 0 ? ~0ull : (uint64_t)rintl(v);
  }
  return t;
}

}  // namespace ds
