// The FP64 operator's interacting pairs as stored values: a product then
// reads S instead of evaluating it.
//
// GB300 issues FP64 at 2 lanes per clock per SM, so evaluating a pair (~20
// FP64 instructions, pair_f64.cu) takes 10 clocks of an SM; the same pair read
// from HBM as an FP64 value and a column index takes 10 or 12 bytes (0.47 or
// 0.56 clocks at the measured rate) and one FP64 FMA (0.5 clocks).  An iterative
// solve multiplies by the same S a hundred times and more, so the first product
// of an operator evaluates every interacting pair once into this list, and all
// products and residuals read it.  Bound then by the FP64 FMA and HBM about
// equally.
//
// Layout: slices of the 32 rows of a sub-tile, entry e of lane l at
// (start + e) * 32 + l, every row its interacting columns in ascending sorted
// order, so a warp's loads of 32 rows' entries are contiguous; 16-bit column
// indices up to 65,536 padded points, else 32-bit.  Rows of a k-d sub-tile have
// similar counts, the padding (never read) is small.
//
// Measured against evaluating the pairs in every product (Jacobi-PCG to 1e-11,
// the list's construction included): 32,768 pixels, exact kernel 1,146 -> 42.8
// ms (47.0 ms on a new operator); 4,096 pixels, table kernel, with the operator
// and a 131,072-point map 63 -> 8.3 ms.
#include <algorithm>

#include <cub/cub.cuh>

#include "ds_device.cuh"
#include "ds_ops.h"
#include "ds_pairhit.cuh"

namespace ds {

namespace {

// The interacting columns of every row: FILL = false counts them (cnt per
// row, the slice's maximum in smax), true writes their indices to cols.  One
// CTA per row tile, one warp per sub-tile; the same FP32 test in both passes.
template <bool FILL, class I>
__global__ void __launch_bounds__(TILE) k_vals_cols(KernelConsts kc, PairArgs a,
                                                    int* __restrict__ cnt,
                                                    long long* __restrict__ smax,
                                                    const long long* __restrict__ start,
                                                    I* __restrict__ cols) {
  __shared__ float4 scol[TILE / 32][SUBTILE];
  const int t = a.row_order[blockIdx.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = t * TILE + threadIdx.x, s = t * (TILE / 32) + warp;
  float3 row;
  const HitFrame frame = hit_frame(kc, a.rx[i], a.ry[i], a.rz[i], row);
  int n = 0;
  I* out = FILL ? cols + start[s] * 32 + lane : nullptr;
  for (int p = a.row_ptr[t]; p < a.row_ptr[t + 1]; ++p) {
    const unsigned m = (a.mask[p] >> (4 * warp)) & 0xFu;
    if (!m) continue;
    for (int cs = 0; cs < TILE / SUBTILE; ++cs) {
      if (!((m >> cs) & 1u)) continue;
      const int j0 = a.cols[p] * TILE + cs * SUBTILE;
      const float3 c = hit_point(frame, a.cx[j0 + lane], a.cy[j0 + lane], a.cz[j0 + lane]);
      __syncwarp();
      scol[warp][lane] = make_float4(c.x, c.y, c.z, 0.f);
      __syncwarp();
      unsigned h = hit_mask(frame, row, scol[warp]);
      if (i >= a.n_rows) h = 0;  // padding rows and columns carry no term
      if (a.n_cols - j0 < SUBTILE) h &= (1u << max(a.n_cols - j0, 0)) - 1u;
      if (FILL) {
        while (h) {
          out[(size_t)n++ * 32] = (I)(j0 + __ffs(h) - 1);
          h &= h - 1;
        }
      } else {
        n += __popc(h);
      }
    }
  }
  if (!FILL) {
    cnt[i] = n;
    const int m = __reduce_max_sync(0xffffffffu, n);
    if (lane == 0) smax[s] = m;
  }
}

// Values of all entries, one thread per entry (every lane busy up to the
// slices' padding): CTA (slice, part), a warp per entry row.
template <int EVAL, class I>
__global__ void __launch_bounds__(TILE) k_vals_eval(KernelConsts kc, PairArgs a,
                                                    const int* __restrict__ cnt,
                                                    const long long* __restrict__ start,
                                                    const I* __restrict__ cols,
                                                    double* __restrict__ val) {
  __shared__ double tf[EVAL == DS_EVAL_TABLE ? TABLE_N : 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (EVAL == DS_EVAL_TABLE) {
    for (int k = tid; k < TABLE_N; k += TILE) tf[k] = a.table[k];
  } else if (tid < 32) {
    tf[tid] = exp2(-(double)tid / 32.0);
  }
  __syncthreads();
  const int s = blockIdx.x, i = s * 32 + lane;
  const double xi = a.rx[i], yi = a.ry[i], zi = a.rz[i];
  const int n = cnt[i], len = (int)(start[s + 1] - start[s]);
  for (int e = blockIdx.y * (TILE / 32) + warp; e < len; e += gridDim.y * (TILE / 32)) {
    if (e >= n) continue;
    const size_t k = (size_t)(start[s] + e) * 32 + lane;
    const int j = cols[k];
    const double dx = xi - a.cx[j], dy = yi - a.cy[j], dz = zi - a.cz[j];
    val[k] = EVAL == DS_EVAL_TABLE ? gp_table_fast(dx, dy, dz, kc, tf)
                                   : g_exact_fast(dx, dy, dz, kc, tf);
  }
}

// out = A v or b - A v from the list, u the column weights of v: W warps per
// slice, warp w taking entries w, w + W, ... of its 32 rows, U of them in
// flight; the warps' sums are added in order.  The dot product with dotv
// goes to alpha as in the evaluating kernel.
template <int EPI, bool DOT, int W, class I>
__global__ void __launch_bounds__(32 * W) k_vals_mv(PairArgs a, const int* __restrict__ cnt,
                                                    const long long* __restrict__ start,
                                                    const I* __restrict__ cols,
                                                    const double* __restrict__ val) {
  if (a.skip_flag && *a.skip_flag) return;
  constexpr int U = 8;
  __shared__ double part[W][32];
  __shared__ double red[W];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // heaviest row tiles first
  const int s = a.row_order[blockIdx.x / (TILE / 32)] * (TILE / 32) + blockIdx.x % (TILE / 32);
  const int i = s * 32 + lane, n = cnt[i];
  const long long s0 = start[s];
  const int len = (int)(start[s + 1] - s0);
  const I* c = cols + s0 * 32 + lane;
  const double* g = val + s0 * 32 + lane;
  double acc = 0.0;
  for (int e = warp; e < len; e += W * U) {
    int j[U];
    double q[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const bool in = e + k * W < n;
      j[k] = in ? (int)__ldcs(c + (size_t)(e + k * W) * 32) : -1;
      q[k] = in ? __ldcs(g + (size_t)(e + k * W) * 32) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (j[k] >= 0) acc = fma(q[k], a.u[j[k]], acc);
  }
  part[warp][lane] = acc;
  __syncthreads();
  if (warp == 0) {
    for (int w = 1; w < W; ++w) acc += part[w][lane];
    const double q = a.wl[i] * acc + a.e[i] * a.v[i];
    const double o = EPI == EPI_RESIDUAL ? a.b[i] - q : q;
    a.out[i] = o;
    if (a.prof_pairs) {
      const int evaluated = __reduce_add_sync(0xffffffffu, n);
      if (lane == 0) atomicAdd(a.prof_pairs, (unsigned long long)evaluated);
    }
    if (DOT) {
      double d = a.dotv[i] * o;
      for (int k = 16; k > 0; k >>= 1) d += __shfl_down_sync(0xffffffffu, d, k);
      if (lane == 0) a.dot_partial[s] = d;
    }
  }
  if (DOT && last_block_arrive(a.counter)) {
    const double dq = reduce_partials<32 * W>(a.dot_partial, gridDim.x, 1, 0, red);
    if (threadIdx.x == 0) {
      a.pcg->dq = dq;
      a.pcg->alpha = a.pcg->delta / dq;  // lib/pcg.h:37
      *a.counter = 0;
    }
  }
}

template <int W, class I>
void launch_mv(int epi, const PairArgs& a, int n_slices, const PairVals& pv, const I* cols,
               cudaStream_t st) {
  if (epi == EPI_RESIDUAL)
    k_vals_mv<EPI_RESIDUAL, false, W, I>
        <<<n_slices, 32 * W, 0, st>>>(a, pv.cnt.p, pv.start.p, cols, pv.val.p);
  else if (a.dot_partial)
    k_vals_mv<EPI_PRODUCT, true, W, I>
        <<<n_slices, 32 * W, 0, st>>>(a, pv.cnt.p, pv.start.p, cols, pv.val.p);
  else
    k_vals_mv<EPI_PRODUCT, false, W, I>
        <<<n_slices, 32 * W, 0, st>>>(a, pv.cnt.p, pv.start.p, cols, pv.val.p);
}

template <int W>
void launch_mv(int epi, const PairArgs& a, int n_slices, const PairVals& pv, cudaStream_t st) {
  if (pv.col16.p)
    launch_mv<W>(epi, a, n_slices, pv, pv.col16.p, st);
  else
    launch_mv<W>(epi, a, n_slices, pv, pv.col32.p, st);
}

template <class I>
void fill(ds_operator* op, PairVals& pv, const PairArgs& a, DevBuf<I>& cols, cudaStream_t st) {
  k_vals_cols<true, I><<<op->pix.n_tiles, TILE, 0, st>>>(op->kc, a, nullptr, nullptr, pv.start.p,
                                                         cols.p);
  DS_CHECK_LAUNCH();
  // enough CTAs for 16 per SM (152) when there are few slices
  const int ns = op->pix.n_pad / 32;
  const dim3 grid(ns, std::max(1, std::min(32, (2432 + ns - 1) / ns)));
  if (vals_fx_usable(op->kc, op->pix)) {
    fill_vals_fx(op, grid, st);
    return;
  }
  if (op->kc.eval == DS_EVAL_TABLE)
    k_vals_eval<DS_EVAL_TABLE, I>
        <<<grid, TILE, 0, st>>>(op->kc, a, pv.cnt.p, pv.start.p, cols.p, pv.val.p);
  else
    k_vals_eval<DS_EVAL_EXACT, I>
        <<<grid, TILE, 0, st>>>(op->kc, a, pv.cnt.p, pv.start.p, cols.p, pv.val.p);
  DS_CHECK_LAUNCH();
}

}  // namespace

size_t store_budget(ds_context* ctx) {
  size_t free_b = 0, total_b = 0;
  DS_CUDA(cudaMemGetInfo(&free_b, &total_b));
  cudaMemPool_t pool;
  DS_CUDA(cudaDeviceGetDefaultMemPool(&pool, ctx->device));
  unsigned long long held = 0, used = 0;
  DS_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held));
  DS_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
  return (size_t)(ctx->store_share * (double)(free_b + (held > used ? held - used : 0)));
}

static void drop_vals(PairVals& pv) {
  pv.ok = false;
  pv.cnt.release();
  pv.start.release();
  pv.val.release();
  pv.col16.release();
  pv.col32.release();
}

bool drop_pair_vals(ds_operator* op) {
  if (!op->vals.ok) return false;
  drop_vals(op->vals);
  op->vals.decided = 0;
  return true;
}

static bool build_vals(ds_operator* op);

// Builds the list on the operator's first product; false when the operator
// evaluates its pairs on every product instead: when the list would take more
// than the context's share (an eighth unless set) of the device memory that is
// free, so that it does not crowd out what the caller allocates later, or when an
// allocation fails.  Decided again when the share is set; share 0 gives the list
// back.
bool ensure_pair_vals(ds_operator* op) {
  PairVals& pv = op->vals;
  if (pv.decided == op->ctx->share_serial) return pv.ok;
  if (!(pv.ok && op->ctx->store_share > 0.0)) {
    drop_vals(pv);
    try {
      pv.ok = op->ctx->store_share > 0.0 && build_vals(op);
    } catch (const Error& e) {
      drop_vals(pv);
      if (e.code != DS_ERR_OOM) throw;
      cudaGetLastError();  // the failed allocation's
    }
    if (!pv.ok) drop_vals(pv);
  }
  pv.decided = op->ctx->share_serial;
  return pv.ok;
}

// Counting pass, scan, indices, values; false when over the budget.
static bool build_vals(ds_operator* op) {
  PairVals& pv = op->vals;
  PairArgs a = op_pair_args(op, nullptr, nullptr);
  cudaStream_t st = op->ctx->stream;
  const int ns = op->pix.n_pad / 32;
  DevBuf<long long> smax;  // ns + 1: the last one 0 for the scan's total
  smax.alloc(ns + 1);
  pv.cnt.alloc(op->pix.n_pad);
  pv.start.alloc(ns + 1);
  DS_CUDA(cudaMemsetAsync(smax.p + ns, 0, sizeof(long long), st));
  k_vals_cols<false, int><<<op->pix.n_tiles, TILE, 0, st>>>(op->kc, a, pv.cnt.p, smax.p, nullptr,
                                                           nullptr);
  DS_CHECK_LAUNCH();
  size_t tmp_bytes = 0;
  DS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, smax.p, pv.start.p, ns + 1, st));
  DevBuf<unsigned char> tmp;
  tmp.alloc(std::max<size_t>(tmp_bytes, 1));
  DS_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tmp_bytes, smax.p, pv.start.p, ns + 1, st));
  long long rows = 0;  // entry rows of 32 entries
  DS_CUDA(cudaMemcpyAsync(&rows, pv.start.p + ns, sizeof(rows), cudaMemcpyDeviceToHost, st));
  DS_CUDA(cudaStreamSynchronize(st));
  const bool narrow = op->pix.n_pad <= 65536;
  const size_t n = (size_t)std::max<long long>(rows, 1) * 32;
  if (n * (narrow ? 10 : 12) > store_budget(op->ctx)) return false;
  pv.val.alloc(n);
  if (narrow) {
    pv.col16.alloc(n);
    fill(op, pv, a, pv.col16, st);
  } else {
    pv.col32.alloc(n);
    fill(op, pv, a, pv.col32, st);
  }
  return true;
}

// a: op_pair_args(op, v, out) (+ dot product arguments); u: the column
// weights of v already formed.
void launch_pair_vals(ds_operator* op, int epi, const PairArgs& a0, cudaStream_t st) {
  PairArgs a = a0;
  cudaEvent_t ev = nullptr;
  a.prof_pairs = nullptr;
  if (a.prof && a.prof->enabled) {
    a.prof_pairs = a.prof->d_pairs;
    a.prof->begin(st, &ev);
  }
  // warps per slice: about 32 resident warps per SM or more
  const int ns = op->pix.n_pad / 32;
  if (ns >= 1216)
    launch_mv<4>(epi, a, ns, op->vals, st);
  else if (ns >= 608)
    launch_mv<8>(epi, a, ns, op->vals, st);
  else
    launch_mv<16>(epi, a, ns, op->vals, st);
  DS_CHECK_LAUNCH();
  if (ev) a.prof->end(st, ev, 0);
}

}  // namespace ds
