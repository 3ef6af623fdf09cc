// FP64 matrix-free pair kernel: one CTA per row tile, one row per thread,
// looping over the row tile's culled column tiles: an FP32 search finds the
// interacting pairs, which alone are evaluated in FP64.  The 200-knot table
// lives in shared memory.  Serves
//   * WFVector{SN,W}::A_product / A_residual (lib/wf_vector.cc:51-103,
//     196-251), with the CG dot d.q fused into the product epilogue;
//   * smp_product (lib/map.cc:20-43);
//   * sigma_m_noise_dom (lib/map_covar.cc:11-38).
// Roofline: FP64 pipe (about 19 FP64 instructions per interacting pair with
// either kernel); no HBM traffic beyond the tiles (L2 resident).
#include <algorithm>

#include "ds_device.cuh"
#include "ds_ops.h"
#include "ds_pairhit.cuh"

namespace ds {

namespace {

// Each warp's 32 rows form a k-d sub-tile with its own box; a column tile is
// four 32-column sub-tiles, and a warp visits only the column sub-tiles whose
// box is within the cutoff of its own (the pair mask).  Per visited block the
// FP32 test (ds_pairhit.cuh) gives every lane the columns that may interact
// with its row; they go to the lane's queue in shared memory, in column
// order, and are evaluated in FP64 from there.  A row's sum takes its
// interacting columns in ascending tile, sub-tile and column order (the terms
// left out are exact zeros).
//
// Bound: the FP64 pipe, ~20 instructions per interacting pair (2 lanes per
// clock per SM).  A queue of QLEN columns per lane is drained only when one
// fills, so a step that evaluates one pair per lane finds almost all lanes
// busy (rows of a sub-tile have similar neighbourhoods, single blocks do
// not).  Measured against evaluating every pair of the visited blocks: the
// 409,600-point exact map of 32,768 pixels 45.0 -> 35.2 ms, the table-kernel
// solve and 131,072-point map of 4,096 pixels 115 -> 63 ms, the same bits.  Where the
// correlation lengths reach the box's size every pair of a block interacts, and the
// queue's 60 clocks a pair (its push loop) are left out: a map of 500 points from 3,000
// pixels 2.54 -> 2.39 ms (2.38 without the search).
constexpr int QLEN = 64;  // a block adds at most 32

template <int EVAL, int EPI, bool DOT>
__global__ void __launch_bounds__(TILE) k_pair_f64(KernelConsts kc, PairArgs a) {
  if (a.skip_flag && *a.skip_flag) return;
  __shared__ float4 scol[TILE / 32][SUBTILE];
  __shared__ int queue[TILE / 32][QLEN][32];
  __shared__ double tf[EVAL == DS_EVAL_TABLE ? TABLE_N : 32];
  __shared__ double red[TILE / 32];
  const int t = a.row_order ? a.row_order[blockIdx.x] : blockIdx.x;  // heaviest tiles first
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int i = t * TILE + tid;
  if (EVAL == DS_EVAL_TABLE) {
    for (int k = tid; k < TABLE_N; k += TILE) tf[k] = a.table[k];
  } else if (tid < 32) {
    tf[tid] = exp2(-(double)tid / 32.0);
  }
  __syncthreads();
  const double xi = a.rx[i], yi = a.ry[i], zi = a.rz[i];
  float3 row;
  const HitFrame frame = hit_frame(kc, xi, yi, zi, row);
  double acc = 0.0;
  int head = 0, tail = 0;  // this lane's queue
  auto add = [&](int j) {
    const double dx = xi - a.cx[j], dy = yi - a.cy[j], dz = zi - a.cz[j];
    double g = EVAL == DS_EVAL_TABLE ? gp_table_fast(dx, dy, dz, kc, tf)
                                     : g_exact_fast(dx, dy, dz, kc, tf);
    if (EPI == EPI_NOISE) g = g * g;
    acc = fma(g, a.u[j], acc);
  };
  auto step = [&] {
    if (head < tail) {
      const int j = queue[warp][head & (QLEN - 1)][lane];
      ++head;
      add(j);
    }
  };
  const int p0 = a.row_ptr[t], p1 = a.row_ptr[t + 1];
  for (int p = p0; p < p1; ++p) {
    const unsigned m = (a.mask[p] >> (4 * warp)) & 0xFu;  // this warp's row sub-tile
    if (!m) continue;
    const int ct = a.cols[p];
    for (int cs = 0; cs < TILE / SUBTILE; ++cs) {
      if (!((m >> cs) & 1u)) continue;
      const int j0 = ct * TILE + cs * SUBTILE;
      const float3 c = hit_point(frame, a.cx[j0 + lane], a.cy[j0 + lane], a.cz[j0 + lane]);
      __syncwarp();
      scol[warp][lane] = make_float4(c.x, c.y, c.z, 0.f);
      __syncwarp();
      unsigned h = hit_mask(frame, row, scol[warp]);
      // a block whose every pair may interact needs no queue when that is empty
      if (a.n_cols - j0 >= SUBTILE &&
          __all_sync(0xffffffffu, (h == 0xffffffffu || i >= a.n_rows) && head == tail)) {
        if (i < a.n_rows) {
#pragma unroll 4
          for (int jj = 0; jj < SUBTILE; ++jj) add(j0 + jj);
          head = tail += SUBTILE;
        }
        continue;
      }
      if (i >= a.n_rows) h = 0;  // padding rows and columns carry no term
      if (a.n_cols - j0 < SUBTILE) h &= (1u << max(a.n_cols - j0, 0)) - 1u;
      while (h) {
        queue[warp][tail & (QLEN - 1)][lane] = j0 + __ffs(h) - 1;
        ++tail;
        h &= h - 1;
      }
      while (__any_sync(0xffffffffu, tail - head > QLEN - SUBTILE)) step();
    }
  }
  while (__any_sync(0xffffffffu, head < tail)) step();
  if (a.prof_pairs) {
    const int evaluated = __reduce_add_sync(0xffffffffu, tail);
    if (lane == 0) atomicAdd(a.prof_pairs, (unsigned long long)evaluated);
  }
  if (EPI == EPI_PRODUCT || EPI == EPI_RESIDUAL) {
    const double q = a.wl[i] * acc + a.e[i] * a.v[i];
    const double o = (EPI == EPI_RESIDUAL) ? a.b[i] - q : q;
    a.out[i] = o;
    if (DOT) {
      const double s = block_sum<TILE>(a.dotv[i] * o, red);
      if (tid == 0) a.dot_partial[t] = s;
      if (last_block_arrive(a.counter)) {
        const double dq = reduce_partials<TILE>(a.dot_partial, gridDim.x, 1, 0, red);
        if (tid == 0) {
          a.pcg->dq = dq;
          a.pcg->alpha = a.pcg->delta / dq;  // lib/pcg.h:37
          *a.counter = 0;
        }
      }
    }
  } else {
    const int dst = a.row_perm[i];
    if (dst >= 0) a.out[dst] = acc;
  }
}

__global__ void k_form_u(int n, double scale, const double* __restrict__ w,
                         const double* __restrict__ v, double* __restrict__ u,
                         const int* skip) {
  if (skip && *skip) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    u[i] = scale * (w ? w[i] * v[i] : v[i]);
}

template <int EVAL>
void launch_eval(const KernelConsts& kc, int epi, const PairArgs& a, cudaStream_t st) {
  const dim3 grid(a.n_row_tiles), block(TILE);
  switch (epi) {
    case EPI_PRODUCT:
      if (a.dot_partial)
        k_pair_f64<EVAL, EPI_PRODUCT, true><<<grid, block, 0, st>>>(kc, a);
      else
        k_pair_f64<EVAL, EPI_PRODUCT, false><<<grid, block, 0, st>>>(kc, a);
      break;
    case EPI_RESIDUAL:
      k_pair_f64<EVAL, EPI_RESIDUAL, false><<<grid, block, 0, st>>>(kc, a);
      break;
    case EPI_MAP:
      k_pair_f64<EVAL, EPI_MAP, false><<<grid, block, 0, st>>>(kc, a);
      break;
    case EPI_NOISE:
      k_pair_f64<EVAL, EPI_NOISE, false><<<grid, block, 0, st>>>(kc, a);
      break;
    default:
      throw Error{DS_ERR_ARG, "bad pair epilogue"};
  }
}

}  // namespace

void form_u(int n_pad, double scale, const double* w, const double* v, double* u,
            const int* skip, cudaStream_t st) {
  k_form_u<<<std::max(1, std::min(1024, (n_pad + 255) / 256)), 256, 0, st>>>(n_pad, scale, w, v, u,
                                                                            skip);
  DS_CHECK_LAUNCH();
}

void launch_pair_f64(const KernelConsts& kc, int epi, const PairArgs& a0, cudaStream_t st,
                     const PointSet* rows, const PointSet* cols) {
  if (a0.n_row_tiles <= 0) return;
  PairArgs a = a0;
  const bool op = epi == EPI_PRODUCT || epi == EPI_RESIDUAL;
  form_u((a.n_cols + TILE - 1) / TILE * TILE, epi == EPI_NOISE ? kc.var_s * kc.var_s : kc.var_s,
         op ? a.wr : nullptr, a.v, a.u, a.skip_flag, st);
  cudaEvent_t ev = nullptr;
  const int kind = epi == EPI_MAP ? 2 : 0;
  if (a.prof && a.prof->enabled) {
    a.prof_pairs = a.prof->d_pairs + kind;
    a.prof->begin(st, &ev);
  } else {
    a.prof_pairs = nullptr;
  }
  if (rows && fx_usable(kc, *rows, *cols))
    launch_pair_fx(kc, epi, a, *rows, *cols, st);
  else if (kc.eval == DS_EVAL_TABLE)
    launch_eval<DS_EVAL_TABLE>(kc, epi, a, st);
  else
    launch_eval<DS_EVAL_EXACT>(kc, epi, a, st);
  DS_CHECK_LAUNCH();
  if (ev) a.prof->end(st, ev, kind);
}

long long& launch_counter() {
  static long long count = 0;
  return count;
}

cudaEvent_t Profiler::get_event() {
  if (!free_events.empty()) {
    cudaEvent_t e = free_events.back();
    free_events.pop_back();
    return e;
  }
  cudaEvent_t e;
  DS_CUDA(cudaEventCreate(&e));
  return e;
}

void Profiler::begin(cudaStream_t st, cudaEvent_t* ev) {
  *ev = get_event();
  DS_CUDA(cudaEventRecord(*ev, st));
}

void Profiler::end(cudaStream_t st, cudaEvent_t start, int kind) {
  cudaEvent_t e = get_event();
  DS_CUDA(cudaEventRecord(e, st));
  pending.push_back(Pending{start, e, kind});
}

void Profiler::collect() {
  // The events go back to the free list before they are read, so that an
  // error thrown from the checks never leaves an event in both lists.
  std::vector<Pending> work;
  work.swap(pending);
  for (const Pending& pr : work) {
    free_events.push_back(pr.start);
    free_events.push_back(pr.stop);
  }
  for (const Pending& pr : work) {
    DS_CUDA(cudaEventSynchronize(pr.stop));
    float t = 0.f;
    DS_CUDA(cudaEventElapsedTime(&t, pr.start, pr.stop));
    ms[pr.kind] += t;
    ++launches[pr.kind];
  }
}

Profiler::~Profiler() {
  for (auto& pr : pending) {
    cudaEventDestroy(pr.start);
    cudaEventDestroy(pr.stop);
  }
  for (auto e : free_events) cudaEventDestroy(e);
  if (d_pairs) cudaFree(d_pairs);
}

}  // namespace ds
