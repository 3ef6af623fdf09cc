// Evaluation of staged columns by the FP32 pair kernels (pair_f32.cu: the
// formulations and the lane layout; persist_pairs.cu), the latter's packing.
#pragma once

#include "ds_f32.h"

namespace ds {

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void kahan_add(float& s, float& c, float v) {
  const float y = v - c;
  const float t = s + y;
  c = (t - s) - y;
  s = t;
}

// A lane's four rows (lane, +32, +64, +96), each coordinate twice: the packed
// operations take one row and two neighbouring columns.  (Two rows and one column, as
// in pair_f32.cu, need the column's four values duplicated into register pairs: 24
// issued instructions a column instead of 15, where 4 exponentials take 16 clocks.
// With 4 warps per scheduler here that is 10.7 -> 9.6 ms a solve at 44,237 pixels; the
// 20 warps per SM of the per-kernel form, at 96 registers, are faster with it: 43.5
// against 45.6 ms at 262,144.)
struct RowRegs {
  float2 x[4], y[4], z[4];
  __device__ __forceinline__ void set(int k, float4 v) {
    x[k] = make_float2(v.x, v.x);
    y[k] = make_float2(v.y, v.y);
    z[k] = make_float2(v.z, v.z);
  }
};

// One warp's 32 staged columns against its lane's four rows, added to acc in column
// order.  Columns 2 p, 2 p + 1 are at col[2 p] = (x, x', y, y') and col[2 p + 1] =
// (z, z', w, w'), their values four to a shared-memory load.  A pair of rows whose
// two row sub-tiles are both beyond the cutoff from the column sub-tile is skipped
// (DO01 / DO23 false).  QU: groups of four columns unrolled.
template <int FORMULA, bool DO01, bool DO23, int QU>
__device__ __forceinline__ void accumulate32(const float4* __restrict__ col,
                                             const float4* __restrict__ cu4, const RowRegs& R,
                                             float (&acc)[4]) {
#pragma unroll QU
  for (int qd = 0; qd < 8; ++qd) {
    const float4 u4 = cu4[qd];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 a = col[4 * qd + 2 * h], b = col[4 * qd + 2 * h + 1];
      const float u0 = h ? u4.z : u4.x, u1 = h ? u4.w : u4.y;
#pragma unroll
      for (int r = DO01 ? 0 : 2; r < (DO23 ? 4 : 2); ++r) {
        float2 t;
        if (FORMULA == F32_EXPANDED) {
          t = __ffma2_rn(R.x[r], make_float2(a.x, a.y), make_float2(b.z, b.w));
          t = __ffma2_rn(R.y[r], make_float2(a.z, a.w), t);
          t = __ffma2_rn(R.z[r], make_float2(b.x, b.y), t);
        } else {  // the columns are staged negated: d = row - column, t = -|d|^2
          const float2 dx = __fadd2_rn(R.x[r], make_float2(a.x, a.y));
          const float2 dy = __fadd2_rn(R.y[r], make_float2(a.z, a.w));
          const float2 dz = __fadd2_rn(R.z[r], make_float2(b.x, b.y));
          t = __fmul2_rn(dx, make_float2(-dx.x, -dx.y));
          t = __ffma2_rn(dy, make_float2(-dy.x, -dy.y), t);
          t = __ffma2_rn(dz, make_float2(-dz.x, -dz.y), t);
        }
        acc[r] = __fmaf_rn(ex2f(t.x), u0, acc[r]);
        acc[r] = __fmaf_rn(ex2f(t.y), u1, acc[r]);
      }
    }
  }
}

// The 32 columns of one staged work item with the row pairs its mask names.
template <int FORMULA, int QU>
__device__ __forceinline__ void accumulate_item(unsigned m, const float4* __restrict__ col,
                                                const float4* __restrict__ cu4,
                                                const RowRegs& R, float (&acc)[4]) {
  const bool do01 = (m & 3u) != 0;   // row sub-tile 0 or 1
  const bool do23 = (m & 12u) != 0;  // row sub-tile 2 or 3
  if (do01 && do23)
    accumulate32<FORMULA, true, true, QU>(col, cu4, R, acc);
  else if (do01)
    accumulate32<FORMULA, true, false, QU>(col, cu4, R, acc);
  else if (do23)
    accumulate32<FORMULA, false, true, QU>(col, cu4, R, acc);
}

// A column to stage: this lane's column (tile-relative), its tile's origin, its
// value and the row sub-tiles that interact with the item's columns (bit k).
struct ColRegs {
  float3 q, o;
  float u;  // colw v (product) or v (map)
  unsigned m;
};

// The column in the frame of the row tile with origin ot.
template <int FORMULA>
__device__ __forceinline__ float4 column_in_frame(const ColRegs& c, const float4& ot) {
  const float dx = ot.x - c.o.x, dy = ot.y - c.o.y, dz = ot.z - c.o.z;
  const float zx = c.q.x - dx, zy = c.q.y - dy, zz = c.q.z - dz;
  if (FORMULA == F32_EXPANDED) {
    const float aj = fmaf(zx, zx, fmaf(zy, zy, zz * zz));
    return make_float4(2.f * zx, 2.f * zy, 2.f * zz, -aj);
  }
  return make_float4(-zx, -zy, -zz, 0.f);
}

// A warp stages its 32 columns (one per lane) at col in accumulate32's layout: the
// even lane of a pair writes the x and y, the odd one z and w.
__device__ __forceinline__ void stage_columns(float4* col, const float4& v) {
  const int lane = threadIdx.x & 31;
  const bool odd = lane & 1;
  const float s0 = __shfl_xor_sync(0xffffffffu, odd ? v.x : v.z, 1);
  const float s1 = __shfl_xor_sync(0xffffffffu, odd ? v.y : v.w, 1);
  col[lane] = odd ? make_float4(s0, v.z, s1, v.w) : make_float4(v.x, s0, v.y, s1);
}

}  // namespace ds
