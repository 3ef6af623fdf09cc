// Dot products of FP32 vectors scaled by powers of two: in float pairs (exact
// products by FMA, compensated sums, about 44 bits) within a warp and FP64 from there
// up, the persistent structured form (persist.cu); in three floats (more bits than
// FP64 sums) within a tile, the batched solve (batch.cu).
#pragma once

#include "ds_f32.h"
#include "ds_ff.cuh"
#include "ds_mixed_dev.cuh"

namespace ds {

// a += x y exactly rounded to a float pair (the product's error by FMA).
__device__ __forceinline__ void ff_acc_prod(ff& a, float x, float y) {
  ff p;
  p.h = __fmul_rn(x, y);
  p.l = __fmaf_rn(x, y, -p.h);
  a = ff_add(a, p);
}

// Sums in three floats: every rounding error of the first is added to the second
// and that sum's to the third, so that a sum of n terms is within n^3 2^-72 of the
// exact one, better than FP64's n 2^-53 up to some 700 terms.
struct f3 {
  float a, b, c;
};

// v += x y (the product's error by FMA).
__device__ __forceinline__ void f3_acc_prod(f3& v, float x, float y) {
  const float p = __fmul_rn(x, y), e = __fmaf_rn(x, y, -p);
  float e1, e2, e3;
  two_sum(v.a, p, v.a, e1);
  two_sum(v.b, e1, v.b, e2);
  two_sum(v.b, e, v.b, e3);
  v.c = __fadd_rn(v.c, __fadd_rn(e2, e3));
}

__device__ __forceinline__ void f3_add(f3& v, const f3& w) {
  float e1, e2, e3;
  two_sum(v.a, w.a, v.a, e1);
  two_sum(v.b, e1, v.b, e2);
  two_sum(v.b, w.b, v.b, e3);
  v.c = __fadd_rn(__fadd_rn(v.c, w.c), __fadd_rn(e2, e3));
}

__device__ __forceinline__ double f3_double(const f3& v) {
  return (double)v.a + ((double)v.b + (double)v.c);
}

__device__ __forceinline__ ff ff_shfl_down(ff v, int o) {
  ff r;
  r.h = __shfl_down_sync(0xffffffffu, v.h, o);
  r.l = __shfl_down_sync(0xffffffffu, v.l, o);
  return r;
}

__device__ __forceinline__ double ff_double(ff v) { return (double)v.h + (double)v.l; }

// Sums over the CTA of one or (TWO) two float pairs per thread, in a fixed order:
// float-pair shuffle trees within the warps, whose sums warp 0 alone adds in FP64 by a
// tree, valid in its lanes 0 and (the second sum) 16.  A dependent FP64 addition takes
// 66 clocks with up to 4 warps of an SM at it but 300 with 16: one warp at it is as
// fast as float pairs (some 20 dependent operations), and keeps 53 bits.
template <int NT, bool TWO>
__device__ __forceinline__ double block_sum2(ff v, ff w, float2* sm /* 2 NT / 32 */) {
  constexpr int W = NT / 32;
  static_assert(W <= 16 && (W & (W - 1)) == 0, "two sums share a warp");
  for (int o = 16; o > 0; o >>= 1) {
    const ff a = ff_shfl_down(v, o);
    if (TWO) w = ff_add(w, ff_shfl_down(w, o));
    v = ff_add(v, a);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    sm[wid] = make_float2(v.h, v.l);
    if (TWO) sm[W + wid] = make_float2(w.h, w.l);
  }
  __syncthreads();
  double s = 0.0;
  if (wid == 0) {
    if ((lane & 15) < W && (TWO || lane < 16)) {
      const float2 t = sm[(lane >> 4) * W + (lane & 15)];
      s = (double)t.x + (double)t.y;
    }
    for (int o = W / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 16);
  }
  return s;
}

// 2^-e within FP32's normal range.
__device__ __forceinline__ float pow2_neg(int e) {
  return __int_as_float((127 - max(-126, min(126, e))) << 23);
}

// The recurrence's scalars between two updates (a MixedState holds them at the ends
// and across updates).  The sums take sr r, sz z, sr q and sz p, powers of two that
// bring |r| and r.z at the last update to about 1 (the squares of vectors in units
// far from 1, fluxes of 1e-17, would leave FP32's range), and stay in those units.
// The norms are kept as squares, with their thresholds, and compared as the integers of
// the same order that the numbers' bits are: they only decide when an update is due, an
// FP64 root takes as long as a dozen additions, and an FP64 instruction of one lane
// holds its scheduler's pipe for 64 clocks.
struct FastState {
  float sr, sz;
  double rz, rz_old, pq;               // times sr sz
  double rr, rrmax, tol2;              // squares, times sr^2 (tol2 < 0: no tolerance)
  double due, half;                    // delta^2 rrmax; a quarter of the best rr
  double delta2, urr;                  // delta^2; 1 / sr^2
  ff alpha;
  float beta;
  int it_best;
};

// The quotient of two FP64 numbers as a float pair (48 bits, what the vectors'
// updates take): long division in two FP32 digits, the remainder of the first in FP64.
__device__ __forceinline__ ff quotient_ff(double a, double b) {
  const float bf = (float)b, q = __fdiv_rn((float)a, bf);
  const float q1 = __fdiv_rn((float)fma(-(double)q, b, a), bf);
  ff r;
  fast_two_sum(q, q1, r.h, r.l);
  return r;
}

// From s, whose residual norm is rnorm.
__device__ __forceinline__ void fast_from(FastState& f, const MixedState& s, double rnorm) {
  const int er = rnorm > 0.0 ? ilogb(rnorm) : 0, ez = s.rz > 0.0 ? ilogb(s.rz) : 0;
  f.sr = pow2_neg(er);
  f.sz = pow2_neg(ez - er);
  const double sr = f.sr, sq = sr * (double)f.sz;
  auto square = [&](double v) { return v * sr * (v * sr); };
  f.rz = s.rz * sq;
  f.rz_old = s.rz_old * sq;
  f.rr = square(rnorm);
  f.rrmax = square(s.rmax);
  f.half = 0.25 * square(s.rbest);
  f.tol2 = s.tol_norm_b >= 0.0 ? square(s.tol_norm_b) : -1.0;
  f.delta2 = s.delta * s.delta;
  f.due = f.delta2 * f.rrmax;
  f.urr = 1.0 / (sr * sr);
  f.beta = (float)s.beta;
  f.it_best = s.it_best;
}

__device__ __forceinline__ void fast_to(const FastState& f, MixedState& s) {
  const double ur = 1.0 / (double)f.sr, uq = 1.0 / ((double)f.sr * (double)f.sz);
  s.rz = f.rz * uq;
  s.rz_old = f.rz_old * uq;
  s.pq = f.pq * uq;
  s.alpha = ff_double(f.alpha);
  s.beta = f.beta;
  s.rnorm = sqrt(f.rr) * ur;
  s.rmax = sqrt(f.rrmax) * ur;
  s.rbest = sqrt(4.0 * f.half) * ur;
  s.it_best = f.it_best;
}

// The step's scalars: of r.z, and of |r|^2 of iteration `it` (the reliable-update
// decision as in update_due).
__device__ __forceinline__ void fast_beta(FastState& f, double trz) {
  f.rz_old = f.rz;
  f.rz = trz;
  f.beta = quotient_ff(trz, f.rz_old).h;
}

__device__ __forceinline__ void fast_norm(FastState& f, MixedState& s, int it, double trr) {
  auto bits = [](double v) { return __double_as_longlong(v); };  // (a NaN: above all)
  f.rr = trr;
  s.iter = it;
  if (bits(trr) > bits(f.rrmax) && bits(trr) <= 0x7ff0000000000000ll) {
    f.rrmax = trr;
    f.due = f.delta2 * trr;
  }
  if (bits(trr) < bits(f.half)) {
    f.half = 0.25 * trr;
    f.it_best = it;
  }
  const bool stall = it - f.it_best >= STALL_ITERS;
  if (stall) s.stalled = 1;
  s.need_update = bits(trr) < bits(f.due) || bits(trr) <= bits(f.tol2) || it >= s.max_iter || stall
                      ? 1
                      : 0;
}

}  // namespace ds
