// Pair sums with the exact kernel in fixed point (ds_fx.cuh): the map and noise
// sums, and the values of the operator's stored pairs.
//
// One CTA per row tile, one row per thread, a warp per 32-row sub-tile, as the
// FP64 kernel (pair_f64.cu).  Per visited 32 x 32 block the FP32 test of
// ds_pairhit.cuh, here on 32-bit integer coordinates, finds the interacting
// pairs; the columns that interact with any of the warp's rows are then
// evaluated for all of them (a value costs ~70 integer instructions, less than
// moving it through a queue), broadcast from shared memory, and the others'
// values are taken as 0.  Sums are FP64 FMAs in the FP64 kernel's order.
//
// Bound: integer issue and the FP64 FMA (0.5 clocks a pair) about equally.
// Measured: the map of 409,600 points and 32,768 pixels 35.2 -> 5.2 ms, the values
// of that operator's stored pairs 2.9 -> 0.6 ms, no larger error.
#include <algorithm>
#include <cmath>

#include "ds_device.cuh"
#include "ds_ops.h"
#include "ds_pairhit.cuh"
#include "fx_tables.h"

namespace ds {

namespace {

struct FxScale {
  double o[3];           // origin
  double hi[3], lo[3];   // sqrt(c) as a double-double
  double coarse;         // 32-bit coordinates per unit
};

// Fixed-point and 32-bit coordinates of n points (see FxPoints).
__global__ void k_fx_points(int n, FxScale f, const double* __restrict__ x,
                            const double* __restrict__ y, const double* __restrict__ z,
                            uint64_t* __restrict__ fx, int4* __restrict__ c) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double v[3] = {x[i], y[i], z[i]};
  int q[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double d = __dsub_rn(v[a], f.o[a]), bb = __dsub_rn(d, v[a]);
    const double err = __dadd_rn(__dsub_rn(v[a], __dsub_rn(d, bb)), __dsub_rn(-f.o[a], bb));
    fx[(size_t)a * n + i] =
        fx_coord(d, err, f.hi[a], f.lo[a], [](double p, double r, double s) { return __fma_rn(p, r, s); },
                 [](double p) { return (int64_t)__double2ll_rn(p); });
    q[a] = __double2int_rn(d * f.hi[a] * f.coarse);
  }
  c[i] = make_int4(q[0], q[1], q[2], 0);
}

struct FxArgs {
  const uint64_t *row, *col;  // three coordinates each, n_row_pad / n_col_pad apart
  size_t n_row, n_col;
  const int4 *rowc, *colc;
  float unit;                 // units per 32-bit coordinate
  float cut;                  // the exponent's cutoff
  uint64_t cut56;             // the same in units of 2^-56
  const uint64_t* tab;        // T1, T2
  int n1;                     // entries of T1 in use
};

__device__ __forceinline__ float3 fx_rel(int4 c, int4 o, float unit) {
  return make_float3((float)(c.x - o.x) * unit, (float)(c.y - o.y) * unit,
                     (float)(c.z - o.z) * unit);
}

// Threshold of the FP32 test: coordinates are off by half a 32-bit unit each
// and by 2^-24 of up to E + S from the conversion (E: largest of the warp's
// rows, S = sqrt(cut)), so a difference by at most d = unit + 2^-22 (E + S) and
// the squared distance of an interacting pair by 2 sqrt(3) S d + 3 d^2.
__device__ __forceinline__ float fx_threshold(const FxArgs& f, const float3& row) {
  float e = fmaxf(fabsf(row.x), fmaxf(fabsf(row.y), fabsf(row.z)));
  for (int o = 16; o > 0; o >>= 1) e = fmaxf(e, __shfl_xor_sync(0xffffffffu, e, o));
  const float s = sqrtf(f.cut), d = f.unit + (e + s) * (1.f / (1 << 22));
  return f.cut * (1.f + 1.f / (1 << 20)) + 4.f * s * d + 4.f * d * d;
}

// exp(-|dX|^2), or 0 at and beyond the cutoff and for pairs that the FP32 test
// left out (whose differences may have wrapped).
__device__ __forceinline__ double fx_value(uint64_t dx, uint64_t dy, uint64_t dz, bool hit,
                                           uint64_t cut56, const uint64_t* t1,
                                           const uint64_t* t2) {
  const uint64_t arg = fx_arg(dx, dy, dz);
  const bool in = hit && arg < cut56;
  const uint64_t bits = fx_exp_bits(in ? arg : 0ull, t1, t2);
  return in ? __longlong_as_double((long long)bits) : 0.0;
}

template <int EPI>
__global__ void __launch_bounds__(TILE) k_pair_fx(FxArgs f, PairArgs a) {
  extern __shared__ __align__(16) uint64_t fsm[];
  uint64_t* t1 = fsm;
  __shared__ uint64_t t2[FX_T2];
  __shared__ ulonglong2 sxy[TILE / 32][SUBTILE];
  __shared__ ulonglong2 szu[TILE / 32][SUBTILE];  // z and the FP64 weight
  __shared__ float4 sc[TILE / 32][SUBTILE];
  const int t = a.row_order[blockIdx.x];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int i = t * TILE + tid;
  for (int k = tid; k < f.n1; k += TILE) t1[k] = f.tab[k];
  for (int k = tid; k < FX_T2; k += TILE) t2[k] = f.tab[FX_T1 + k];
  __syncthreads();
  const uint64_t X = f.row[i], Y = f.row[f.n_row + i], Z = f.row[2 * f.n_row + i];
  const int4 c0 = f.rowc[t * TILE + 32 * warp];  // the warp's frame: its first row
  const float3 row = fx_rel(f.rowc[i], c0, f.unit);
  HitFrame frame;
  frame.thr = fx_threshold(f, row);
  double acc = 0.0;
  unsigned evaluated = 0;
  const int p1 = a.row_ptr[t + 1];
  for (int p = a.row_ptr[t]; p < p1; ++p) {
    const unsigned m = (a.mask[p] >> (4 * warp)) & 0xFu;  // this warp's row sub-tile
    if (!m) continue;
    const int ct = a.cols[p];
    for (int cs = 0; cs < TILE / SUBTILE; ++cs) {
      if (!((m >> cs) & 1u)) continue;
      const int j0 = ct * TILE + cs * SUBTILE, j = j0 + lane;
      const float3 c = fx_rel(f.colc[j], c0, f.unit);
      const ulonglong2 xy = make_ulonglong2(f.col[j], f.col[f.n_col + j]);
      const ulonglong2 zu = make_ulonglong2(
          f.col[2 * f.n_col + j], (unsigned long long)__double_as_longlong(a.u[j]));
      __syncwarp();
      sc[warp][lane] = make_float4(c.x, c.y, c.z, 0.f);
      sxy[warp][lane] = xy;
      szu[warp][lane] = zu;
      __syncwarp();
      unsigned h = hit_mask(frame, row, sc[warp]);
      if (i >= a.n_rows) h = 0;  // padding rows and columns carry no term
      if (a.n_cols - j0 < SUBTILE) h &= (1u << max(a.n_cols - j0, 0)) - 1u;
      evaluated += __popc(h);
      unsigned any = __reduce_or_sync(0xffffffffu, h);
      while (any) {
        const int jj = __ffs(any) - 1;
        any &= any - 1;
        const ulonglong2 q = sxy[warp][jj], w = szu[warp][jj];
        double g = fx_value(X - q.x, Y - q.y, Z - w.x, (h >> jj) & 1u, f.cut56, t1, t2);
        if (EPI == EPI_NOISE) g = g * g;
        acc = fma(g, __longlong_as_double((long long)w.y), acc);
      }
    }
  }
  if (a.prof_pairs) {
    const unsigned n = __reduce_add_sync(0xffffffffu, evaluated);
    if (lane == 0) atomicAdd(a.prof_pairs, (unsigned long long)n);
  }
  const int dst = a.row_perm[i];
  if (dst >= 0) a.out[dst] = acc;
}

// Values of the stored pairs, as k_vals_eval (pair_vals.cu): one thread per
// entry.  A pair of the list that passed the FP32 test without interacting lies
// beyond the cutoff by less than the test's margin (vals_fx_usable).
template <class I>
__global__ void __launch_bounds__(TILE) k_vals_fx(FxArgs f, const int* __restrict__ cnt,
                                                  const long long* __restrict__ start,
                                                  const I* __restrict__ cols,
                                                  double* __restrict__ val) {
  extern __shared__ __align__(16) uint64_t fsm[];
  uint64_t* t1 = fsm;
  __shared__ uint64_t t2[FX_T2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int k = tid; k < f.n1; k += TILE) t1[k] = f.tab[k];
  for (int k = tid; k < FX_T2; k += TILE) t2[k] = f.tab[FX_T1 + k];
  __syncthreads();
  const int s = blockIdx.x, i = s * 32 + lane;
  const uint64_t X = f.row[i], Y = f.row[f.n_row + i], Z = f.row[2 * f.n_row + i];
  const int n = cnt[i], len = (int)(start[s + 1] - start[s]);
  for (int e = blockIdx.y * (TILE / 32) + warp; e < len; e += gridDim.y * (TILE / 32)) {
    if (e >= n) continue;
    const size_t k = (size_t)(start[s] + e) * 32 + lane;
    const int j = cols[k];
    val[k] = fx_value(X - f.col[j], Y - f.col[f.n_col + j], Z - f.col[2 * f.n_col + j], true,
                      f.cut56, t1, t2);
  }
}

FxScale fx_scale(const KernelConsts& kc, const double* lo, const double* hi) {
  FxScale f;
  const double c[3] = {kc.c_perp, kc.c_perp, kc.c_para};
  double ext = 1.0;
  for (int a = 0; a < 3; ++a) {
    f.hi[a] = std::sqrt(c[a]);
    // (0 for an infinite correlation length)
    f.lo[a] = f.hi[a] > 0.0 ? std::fma(-f.hi[a], f.hi[a], c[a]) / (2.0 * f.hi[a]) : 0.0;
    f.o[a] = 0.5 * lo[a] + 0.5 * hi[a];
    ext = std::max(ext, (hi[a] - lo[a]) * f.hi[a]);
  }
  f.coarse = std::ldexp(1.0, 29 - (int)std::ceil(std::log2(ext)));
  return f;
}

void fx_points(FxPoints& p, const FxScale& f, const PointSet& ps, cudaStream_t st) {
  p.fx.alloc((size_t)ps.n_pad * 3);
  p.c.alloc(ps.n_pad);
  k_fx_points<<<(ps.n_pad + 255) / 256, 256, 0, st>>>(
      ps.n_pad, f, ps.x.p, ps.y.p, ps.z.p, reinterpret_cast<uint64_t*>(p.fx.p), p.c.p);
  DS_CHECK_LAUNCH();
}

// Fills the arguments that do not depend on the points; copies the tables.
FxArgs fx_args(const KernelConsts& kc, const FxScale& s, DevBuf<unsigned long long>& tab,
               cudaStream_t st) {
  static const std::vector<uint64_t> t = fx_tables();  // constant; lives with the process
  tab.alloc(t.size());
  DS_CUDA(cudaMemcpyAsync(tab.p, t.data(), tab.bytes(), cudaMemcpyHostToDevice, st));
  FxArgs f{};
  f.unit = (float)(1.0 / s.coarse);
  f.cut = (float)(kc.exact_cut * (1.0 + 1e-6));
  f.cut56 = (uint64_t)std::ceil(std::ldexp(kc.exact_cut, 56));
  f.tab = reinterpret_cast<const uint64_t*>(tab.p);
  f.n1 = std::min(FX_T1, (int)std::ceil(kc.exact_cut * 32.0) + 1);
  return f;
}

void fx_set(FxArgs& f, const FxPoints& rows, const FxPoints& cols) {
  f.row = reinterpret_cast<const uint64_t*>(rows.fx.p);
  f.col = reinterpret_cast<const uint64_t*>(cols.fx.p);
  f.n_row = rows.c.n;
  f.n_col = cols.c.n;
  f.rowc = rows.c.p;
  f.colc = cols.c.p;
}

}  // namespace

// Fixed point needs differences of interacting points below 8 units, with the
// FP32 test's margin (cutoff 48: 6.93 and at most 0.02 of margin), and 32-bit
// coordinates at least 2^-13 fine (extent 2^16 correlation lengths); FP64
// evaluates what lies outside.
bool fx_usable(const KernelConsts& kc, const PointSet& rows, const PointSet& cols) {
  if (kc.eval != DS_EVAL_EXACT || !(kc.exact_cut <= FX_MAX_CUT)) return false;
  const double s[3] = {std::sqrt(kc.c_perp), std::sqrt(kc.c_perp), std::sqrt(kc.c_para)};
  for (int a = 0; a < 3; ++a) {
    const double ext =
        (std::max(rows.hi[a], cols.hi[a]) - std::min(rows.lo[a], cols.lo[a])) * s[a];
    if (!(ext <= 65536.0)) return false;
  }
  return true;
}

// The list's values besides: its search (ds_pairhit.cuh) must not pass pairs from
// beyond the fixed-point range, whose differences wrap.  With a threshold in use
// everywhere (hit_ok, E + S < 2^20 S for E the extent) a pair that passes has |dX|^2
// at most 2^-18 S (2^16 + S) + 2^-18 cut above the cutoff, below 50 at 48.
bool vals_fx_usable(const KernelConsts& kc, const PointSet& ps) {
  if (!kc.hit_ok || !fx_usable(kc, ps, ps)) return false;
  const double s[3] = {std::sqrt(kc.c_perp), std::sqrt(kc.c_perp), std::sqrt(kc.c_para)};
  for (int a = 0; a < 3; ++a)
    if (!((ps.hi[a] - ps.lo[a]) * s[a] < 0x1p19 * std::sqrt(kc.cull_arg))) return false;
  return true;
}

// EPI_MAP and EPI_NOISE of launch_pair_f64 in fixed point (a.u formed).
void launch_pair_fx(const KernelConsts& kc, int epi, const PairArgs& a, const PointSet& rows,
                    const PointSet& cols, cudaStream_t st) {
  double lo[3], hi[3];
  for (int c = 0; c < 3; ++c) {
    lo[c] = std::min(rows.lo[c], cols.lo[c]);
    hi[c] = std::max(rows.hi[c], cols.hi[c]);
  }
  const FxScale s = fx_scale(kc, lo, hi);
  FxPoints pr, pc;  // freed in stream order
  DevBuf<unsigned long long> tab;
  fx_points(pr, s, rows, st);
  fx_points(pc, s, cols, st);
  FxArgs f = fx_args(kc, s, tab, st);
  fx_set(f, pr, pc);
  const size_t smem = (size_t)f.n1 * sizeof(uint64_t);
  if (epi == EPI_MAP)
    k_pair_fx<EPI_MAP><<<a.n_row_tiles, TILE, smem, st>>>(f, a);
  else
    k_pair_fx<EPI_NOISE><<<a.n_row_tiles, TILE, smem, st>>>(f, a);
  DS_CHECK_LAUNCH();
}

// The values of the operator's stored pairs (columns filled).
void fill_vals_fx(ds_operator* op, const dim3& grid, cudaStream_t st) {
  PairVals& pv = op->vals;
  const FxScale s = fx_scale(op->kc, op->pix.lo, op->pix.hi);
  FxPoints p;
  DevBuf<unsigned long long> tab;
  fx_points(p, s, op->pix, st);
  FxArgs f = fx_args(op->kc, s, tab, st);
  fx_set(f, p, p);
  const size_t smem = (size_t)f.n1 * sizeof(uint64_t);
  if (pv.col16.p)
    k_vals_fx<<<grid, TILE, smem, st>>>(f, pv.cnt.p, pv.start.p, pv.col16.p, pv.val.p);
  else
    k_vals_fx<<<grid, TILE, smem, st>>>(f, pv.cnt.p, pv.start.p, pv.col32.p, pv.val.p);
  DS_CHECK_LAUNCH();
}

}  // namespace ds
