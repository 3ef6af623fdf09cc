// The exact kernel exp(-|dX|^2) of two scaled points in 64-bit fixed point, on
// the integer pipe.
//
// GB300 issues FP64 at 2 lanes per clock per SM and 32-bit integer
// multiply-adds at 32 times that and more: a pair value takes ~20 FP64
// instructions (10 clocks of an SM) or ~70 integer ones (~1.1 clocks), and
// fixed point keeps more bits than FP64 on the way:
//  * coordinates scaled by sqrt(c) are held in units of 2^-60, modulo 2^64
//    (formed once per point in double-double arithmetic); a difference of two
//    interacting points is below 8 and exact to the coordinates' 2^-61;
//  * the squared distance in units of 2^-56 (two 32-bit halves, the low-low
//    products dropped: below 3 units);
//  * exp by two tables, 2^-5 and 2^-12 apart, and a cubic on the rest (below
//    2^-12), all to about 2^-55 relative, rounded once to FP64.
// Largest error of a pair value: 1.55e-16 relative for arguments up to 48 and
// coordinates up to 1e5 (tests/cpp/fx_check.cc runs these functions on the
// host), against 4e-16 for exp_neg_f64 and up to 48 x 3 x 1.1e-16 from the FP64
// argument's roundings on top of it.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define DS_FX __host__ __device__ __forceinline__
#else
#define DS_FX static inline
#endif

namespace ds {

constexpr double FX_MAX_CUT = 48.0;   // of the exponent: |dX| stays below 8
constexpr int FX_T1 = 48 * 32 + 1;    // exp(-j / 32)
constexpr int FX_T2 = 128;            // exp(-i / 4096)
constexpr int FX_EXP_BITS = 7;        // low bits of a T1 entry: its exponent

// (x y) >> 32 of two 32-bit numbers
DS_FX uint32_t fx_mulhi32(uint32_t x, uint32_t y) { return (uint32_t)(((uint64_t)x * y) >> 32); }

// (x y) >> 64, low by at most 2
DS_FX uint64_t fx_mulhi64(uint64_t x, uint64_t y) {
  const uint32_t xh = (uint32_t)(x >> 32), xl = (uint32_t)x;
  const uint32_t yh = (uint32_t)(y >> 32), yl = (uint32_t)y;
  return (uint64_t)xh * yh + (((uint64_t)xh * yl) >> 32) + (((uint64_t)xl * yh) >> 32);
}

// |dX|^2 in units of 2^-56 of a difference in units of 2^-60 (|dX| < 8 per
// axis, |dX|^2 < 64).
DS_FX uint64_t fx_arg(uint64_t dx, uint64_t dy, uint64_t dz) {
  const int32_t ax = (int32_t)(dx >> 32), ay = (int32_t)(dy >> 32), az = (int32_t)(dz >> 32);
  const int32_t bx = (int32_t)((uint32_t)dx >> 1), by = (int32_t)((uint32_t)dy >> 1),
                bz = (int32_t)((uint32_t)dz >> 1);
  const int64_t hi = (int64_t)ax * ax + (int64_t)ay * ay + (int64_t)az * az;
  const int64_t lo = (int64_t)ax * bx + (int64_t)ay * by + (int64_t)az * bz;
  return (uint64_t)(hi + (lo >> 30));
}

// The bits of the FP64 exp(-arg), arg in units of 2^-56 below FX_MAX_CUT.
DS_FX uint64_t fx_exp_bits(uint64_t arg, const uint64_t* t1, const uint64_t* t2) {
  const uint32_t hi = (uint32_t)(arg >> 32);
  const uint64_t m1 = t1[hi >> 19], m2 = t2[(hi >> 12) & (FX_T2 - 1)];
  // e = 1 - exp(-r) = r - r^2 (1/2 - r/6 + r^2/24), r the low 44 bits
  const uint64_t r = arg & ((1ull << 44) - 1);
  const uint32_t r32 = (uint32_t)(r >> 12);
  const uint32_t rr = fx_mulhi32(r32, r32);
  const uint32_t h = 0x80000000u - fx_mulhi32(r32, 174763u) + fx_mulhi32(rr, 11u);
  const uint64_t e = r - fx_mulhi32(rr, h);
  uint64_t p = fx_mulhi64(m1, m2);
  p -= fx_mulhi64(p, e << 8);
  // p / 2^62 in (0.96, 2), times 2^-ex
  uint32_t ex = (uint32_t)m1 & ((1u << FX_EXP_BITS) - 1);
  const uint32_t lz = 1u ^ (uint32_t)(p >> 62);
  p <<= lz;
  ex += lz;
  return ((p + 512) >> 10) + ((uint64_t)(1022u - ex) << 52);
}

// One scaled coordinate v = (x - o) (s_hi + s_lo) in units of 2^-60 modulo 2^64,
// x - o as the exact pair (d, derr).
template <class Fma, class Rint>
DS_FX uint64_t fx_coord(double d, double derr, double s_hi, double s_lo, Fma fma_, Rint to_ll) {
  const double p = d * s_hi;
  const double e = fma_(d, s_hi, -p) + (derr * s_hi + d * s_lo);
  const double two60 = 1152921504606846976.0, two64 = 18446744073709551616.0;
  const double q = p * two60;
  // q modulo 2^64, to within +-2^63 (exact: both are multiples of q's ulp)
  const double k = (double)to_ll(q * 0x1p-64);
  return (uint64_t)to_ll(fma_(-k, two64, q)) + (uint64_t)to_ll(e * two60);
}

}  // namespace ds
