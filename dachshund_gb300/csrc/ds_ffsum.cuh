// Sums and CG scalars of the mixed-precision solves in float pairs: the persistent
// structured form (persist.cu) and the batched solve's vector sums (batch.cu).
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

__device__ __forceinline__ ff ff_shfl_down(ff v, int o, int width = 32) {
  ff r;
  r.h = __shfl_down_sync(0xffffffffu, v.h, o, width);
  r.l = __shfl_down_sync(0xffffffffu, v.l, o, width);
  return r;
}

// Sums over the CTA of two float pairs per thread (float-pair shuffle trees, a
// fixed order), valid in lanes 0 and 16 of warp 0.  The Krylov vectors' dot
// products are summed this way from the threads to the grid (exact products by
// FMA, compensated sums, about 44 bits): a dependent FP64 addition takes 300
// clocks with the SM's 16 warps at it (66 with 4), and the FP64 sums and scalars
// of a persistent iteration took 14,000 of its 22,000 clocks at 16 CTAs.
template <int NT>
__device__ __forceinline__ ff block_sum2_ff(ff v, ff w, float2* sm /* 2 NT / 32 */) {
  constexpr int W = NT / 32;
  static_assert(W <= 16 && (W & (W - 1)) == 0, "two sums share a warp");
  for (int o = 16; o > 0; o >>= 1) {
    const ff a = ff_shfl_down(v, o), b = ff_shfl_down(w, o);
    v = ff_add(v, a);
    w = ff_add(w, b);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    sm[wid] = make_float2(v.h, v.l);
    sm[W + wid] = make_float2(w.h, w.l);
  }
  __syncthreads();
  ff s{0.f, 0.f};
  if (wid == 0) {
    if ((lane & 15) < W) {
      const float2 t = sm[(lane >> 4) * W + (lane & 15)];
      s = ff{t.x, t.y};
    }
    for (int o = W / 2; o > 0; o >>= 1) s = ff_add(s, ff_shfl_down(s, o, 16));
  }
  return s;
}

// Sum of n float-pair partials by one warp (valid in lane 0), the same in every
// CTA: lane l takes l, l + 32, ..., then a shuffle tree.
__device__ __forceinline__ ff warp_total_ff(const double* part, int n) {
  ff v{0.f, 0.f};
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += 32) {
    const float2 t = __ldcg(reinterpret_cast<const float2*>(part) + i);
    v = ff_add(v, ff{t.x, t.y});
  }
  for (int o = 16; o > 0; o >>= 1) v = ff_add(v, ff_shfl_down(v, o));
  return v;
}

// The same for n pairs of float pairs.
__device__ __forceinline__ void warp_total2_ff(const double* part, int n, ff& v, ff& w) {
  v = w = ff{0.f, 0.f};
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += 32) {
    const float4 t = __ldcg(reinterpret_cast<const float4*>(part) + i);
    v = ff_add(v, ff{t.x, t.y});
    w = ff_add(w, ff{t.z, t.w});
  }
  for (int o = 16; o > 0; o >>= 1) {
    const ff a = ff_shfl_down(v, o), b = ff_shfl_down(w, o);
    v = ff_add(v, a);
    w = ff_add(w, b);
  }
}

// a / b as a float pair (the quotient of the heads and its correction).
__device__ __forceinline__ ff ff_div(ff a, ff b) {
  const float q = __fdiv_rn(a.h, b.h);
  const float p = __fmul_rn(q, b.h), pe = __fmaf_rn(q, b.h, -p);
  float e = __fsub_rn(__fsub_rn(a.h, p), pe);  // a.h - q b.h (a.h - p is exact)
  e = __fadd_rn(e, __fmaf_rn(-q, b.l, a.l));
  ff r;
  fast_two_sum(q, __fdiv_rn(e, b.h), r.h, r.l);
  return r;
}

__device__ __forceinline__ void store_part(double* part, ff v) {
  *reinterpret_cast<float2*>(part) = make_float2(v.h, v.l);
}

__device__ __forceinline__ double ff_double(ff v) { return (double)v.h + (double)v.l; }

__device__ __forceinline__ void fast_from(FastState& f, const MixedState& s) {
  const double sr = f.sr, sq = sr * (double)f.sz;
  f.rz = ff_from_double(s.rz * sq);
  f.rz_old = ff_from_double(s.rz_old * sq);
  f.beta = (float)s.beta;
  f.rnorm = (float)(s.rnorm * sr);
  f.rmax = (float)(s.rmax * sr);
  f.rbest = (float)(s.rbest * sr);
  f.delta = (float)s.delta;
  f.tol = (float)(s.tol_norm_b * sr);
  f.it_best = s.it_best;
}

// 2^-e within FP32's normal range.
__device__ __forceinline__ float pow2_neg(int e) {
  return __int_as_float((127 - max(-126, min(126, e))) << 23);
}

// The solve's scales, from |r| and r.z at its start, and the scalars.
__device__ __forceinline__ void fast_init(FastState& f, const MixedState& s) {
  const int er = s.rnorm > 0.0 ? ilogb(s.rnorm) : 0, ez = s.rz > 0.0 ? ilogb(s.rz) : 0;
  f.sr = pow2_neg(er);
  f.sz = pow2_neg(ez - er);
  fast_from(f, s);
}

__device__ __forceinline__ void fast_to(const FastState& f, MixedState& s) {
  const double ur = 1.0 / (double)f.sr, uq = 1.0 / ((double)f.sr * (double)f.sz);
  s.rz = ff_double(f.rz) * uq;
  s.rz_old = ff_double(f.rz_old) * uq;
  s.alpha = ff_double(f.alpha);
  s.pq = ff_double(f.pq) * uq;
  s.beta = f.beta;
  s.rnorm = f.rnorm * ur;
  s.rmax = f.rmax * ur;
  s.rbest = f.rbest * ur;
  s.it_best = f.it_best;
}

// |r|^2 into the history.
__device__ __forceinline__ void store_hist(double* hist, const FastState& f, double rr) {
  store_part(hist, ff_from_double(rr * (double)f.sr * (double)f.sr));
}

// The step's scalars of iteration `it` (reliable-update decision as in
// update_due); |sr r|^2 goes to the history as a float pair (hist null:
// nowhere), whose root is taken after the solve (launch_hist_roots).
__device__ __forceinline__ void fast_step(FastState& f, MixedState& s, double* hist,
                                          int it, ff trz, ff trr) {
  f.rz_old = f.rz;
  f.rz = trz;
  f.rnorm = sqrtf(trr.h);
  s.iter = it;
  if (hist) store_part(hist + it, trr);
  f.rmax = fmaxf(f.rmax, f.rnorm);
  if (f.rnorm < 0.5f * f.rbest) {
    f.rbest = f.rnorm;
    f.it_best = it;
  }
  const bool stall = it - f.it_best >= STALL_ITERS;
  if (stall) s.stalled = 1;
  s.need_update =
      f.rnorm < f.delta * f.rmax || f.rnorm <= f.tol || it >= s.max_iter || stall ? 1 : 0;
  f.beta = ff_div(f.rz, f.rz_old).h;
}

}  // namespace ds
