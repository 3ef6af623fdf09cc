// FP32 search for the interacting pairs of a 32-row x 32-column block.
//
// GB300 issues FP64 at 2 lanes per clock per SM (one warp instruction per 64
// clocks of a scheduler), FP32 at 128.  The culled 32 x 32 sub-tile blocks
// hold mostly pairs beyond the cutoff (of the evaluated pairs about one in
// nine interacts with the table kernel, one in three with the exact one), so
// the FP64 kernels first find the interacting pairs in FP32 (~9 instructions
// per pair) and evaluate only those.
//
// The test never misses an interacting pair: coordinates are taken relative
// to one of the warp's rows in FP64, then scaled and rounded to FP32, so for
// an interacting pair every scaled coordinate is at most E + S (E: largest of
// the warp's rows, S = sqrt(cutoff)) with a relative error below 2^-22, and
// the squared distance is off by less than 2^-18 (cutoff + S (E + S)), which
// the threshold adds; beyond E + S = 2^20 S every pair passes, and so does a
// pair whose test overflows to NaN.  The scales are FP64 roots rounded once (a
// coefficient of lengths beyond 1e19 units is subnormal in FP32); where a scale lies
// outside 2^-100 .. 2^100 its power of two multiplies the coordinates in FP64 first,
// so that no interacting pair's leave FP32's range; with a cutoff outside 2^-20 ..
// 2^40 every pair passes (make_consts).  A pair that passes without interacting costs
// one evaluation that gives zero.
#pragma once

#include <cuda_runtime.h>

#include "ds_internal.cuh"

namespace ds {

// One warp's reference frame: a row's coordinates, the scales and the
// threshold (warp-uniform).
struct HitFrame {
  double ox, oy, oz, up, uq;
  float sp, sq, thr;
  int units;
};

__device__ __forceinline__ float3 hit_point(const HitFrame& f, double x, double y, double z) {
  double dx = x - f.ox, dy = y - f.oy, dz = z - f.oz;
  if (f.units) {
    dx *= f.up;
    dy *= f.up;
    dz *= f.uq;
  }
  return make_float3((float)dx * f.sp, (float)dy * f.sp, (float)dz * f.sq);
}

// The frame of the warp's 32 rows (every lane its own row's coordinates) and
// the row's scaled coordinates.
__device__ __forceinline__ HitFrame hit_frame(const KernelConsts& k, double x, double y, double z,
                                              float3& row) {
  constexpr unsigned full = 0xffffffffu;
  HitFrame f;
  f.ox = __shfl_sync(full, x, 0);
  f.oy = __shfl_sync(full, y, 0);
  f.oz = __shfl_sync(full, z, 0);
  f.sp = k.hit_perp;
  f.sq = k.hit_para;
  f.up = k.unit_perp;
  f.uq = k.unit_para;
  f.units = k.hit_units;
  row = hit_point(f, x, y, z);
  float e = fmaxf(fabsf(row.x), fmaxf(fabsf(row.y), fabsf(row.z)));
  for (int o = 16; o > 0; o >>= 1) e = fmaxf(e, __shfl_xor_sync(full, e, o));
  const float cut = __double2float_ru(k.cull_arg), s = sqrtf(cut);
  const float eps = 1.f / (1 << 18);
  f.thr = k.hit_ok && e + s < (float)(1 << 20) * s ? cut + eps * (cut + s * (e + s)) : INFINITY;
  return f;
}

// Bit jj: column jj of the staged block may interact with this lane's row.
__device__ __forceinline__ unsigned hit_mask(const HitFrame& f, const float3& row,
                                             const float4* __restrict__ cols) {
  unsigned m = 0;
#pragma unroll
  for (int jj = 0; jj < SUBTILE; ++jj) {
    const float4 c = cols[jj];
    const float dx = row.x - c.x, dy = row.y - c.y, dz = row.z - c.z;
    const float t = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    if (!(t > f.thr)) m |= 1u << jj;
  }
  return m;
}

}  // namespace ds
