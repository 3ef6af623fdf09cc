// FP32 matrix-free pair kernels of the mixed-precision form: the exact
// kernel var_s exp(-arg) evaluated as var_s 2^(-|dX|^2) on coordinates scaled
// by sqrt(c log2 e), with MUFU ex2 and packed f32x2 FMAs.
//
// Coordinates are stored relative to their tile's origin (the bounding-box
// centre, rounded to FP32), so FP32 differences are taken between numbers of
// the size of a tile rather than of the box.  For a (row tile R, column tile
// C) pair the columns are moved into R's frame once at staging:
//   zeta_j = xi_j - (o_R - o_C).
// Two formulations of the exponent:
//   EXPANDED  t_ij = 2 xi_i . zeta_j - |zeta_j|^2 = |xi_i|^2 - |xi_i - zeta_j|^2,
//             e_ij = 2^t_ij = 2^(|xi_i|^2) S'_ij, the row factor 2^-|xi_i|^2
//             applied once at the end.  Per pair: 3 FFMA + 1 ex2 + 1 FFMA,
//             i.e. 4 FMA-pipe lanes and 1 MUFU: FMA and MUFU (both 32/clk/SM
//             on GB300) are co-bound at 32 pairs/clk/SM.  Relative error of
//             S' about |zeta|^2 * 2^-24 (~1e-6): used for the inner solve,
//             whose FP64 outer residual removes it.
//   DIRECT    t_ij = -|xi_i - zeta_j|^2: 3 FADD + FMUL + 2 FFMA + ex2 + FFMA,
//             7 FMA-pipe lanes (18 pairs/clk/SM); relative error ~1e-7.  Used
//             for the map product and when a tile is too large for EXPANDED
//             (2^|xi|^2 would leave FP32 range).
// Each CTA owns a 128-row tile; lane l of each warp holds rows l, l+32, l+64,
// l+96 (as two f32x2 pairs), and the warps share out the row tile's work
// items (32-column sub-tiles of its interacting column tiles), staging two
// items per round, so a staged column is read once per 4 rows.  Each round's
// FP32 sums (64 terms; 32 for the map, which folds each item on its own) are
// folded into Kahan-compensated FP32 accumulators; the four warps' partial
// rows are summed in FP64 at the end.
#include "ds_device.cuh"
#include "ds_f32.h"
#include "ds_pair_f32.cuh"

namespace ds {

namespace {

// CTAs per SM the register budget is sized for (4 warps each): 96 registers
// hold the two prefetched column tiles and a fully unrolled 32-column loop;
// on the 262,144-pixel workload 5 CTAs per SM beat 4, 6, 7 (with spills) and
// the one-tile prefetch at 8.
constexpr int F32_MIN_CTAS = 5;
constexpr int F32_QU = 2;  // groups of four columns unrolled

template <int FORMULA, int EPI, bool DOT>
__global__ void __launch_bounds__(TILE, F32_MIN_CTAS) k_pair_f32(F32Args a) {
  if (a.skip_flag && *a.skip_flag) return;
  // per warp: two staged work items (64 columns) and their column values
  __shared__ float4 sc[2 * TILE];
  __shared__ float4 su4[2 * TILE / 4];
  __shared__ float sred[4][TILE];
  __shared__ double red[TILE / 32];
  const int t = a.row_order ? a.row_order[blockIdx.x] : blockIdx.x;  // heaviest tiles first
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int base = t * TILE;

  RowRegs R;
#pragma unroll
  for (int k = 0; k < 4; ++k) R.set(k, a.rxi[base + lane + 32 * k]);
  const float4 ot = a.rorig[t];
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  float c0 = 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f;
  unsigned evaluated = 0;  // pairs this warp evaluates (profiling; < 2^32 per warp)

  // Work items (column tile, column sub-tile w) of this row tile, in the
  // order of the tile pairs and then w (build_slice_items); warp v takes
  // items v, v + 4, v + 8, ...: the four warps carry equal work whatever the
  // masks (each warp sums all 128 rows, so the sub-tiles may be shared out
  // freely) and the order of every FP32 sum is fixed.  A warp reads its next
  // 32 items in one load (lane l: its item 32 b + l, the next batch
  // prefetched).  A round stages two items (64 columns, one per lane and
  // item) and folds them into the compensated sums once; the column inputs
  // of the next round are loaded into registers while a round is computed.
  const int i1 = a.item_ptr[t + 1];
  auto load = [&](ColRegs& c, unsigned it) {
    const int ct = (int)(it >> 6);
    const int j = ct * TILE + 32 * (int)((it >> 4) & 3u) + lane;
    const float4 o = a.corig[ct], q = a.cxi[j];
    c.o = make_float3(o.x, o.y, o.z);
    c.q = make_float3(q.x, q.y, q.z);
    c.u = (EPI == EPI_PRODUCT) ? a.colw[j] * a.v[j] : a.v[j];
    c.m = it & 15u;
  };
  constexpr unsigned full = 0xffffffffu;
  int nb = a.item_ptr[t] + warp;  // this warp's first item of the next batch
  unsigned nitem = nb + 4 * lane < i1 ? a.items[nb + 4 * lane] : 0u;
  unsigned witem = 0;  // this lane's item of the current batch
  int pos = 0, cnt = 0;  // items taken / held of the current batch
  auto fetch = [&](ColRegs& c) -> bool {
    if (pos == cnt) {
      if (nb >= i1) return false;
      cnt = min(32, (i1 - nb + 3) >> 2);
      pos = 0;
      witem = nitem;
      nb += 128;
      nitem = nb + 4 * lane < i1 ? a.items[nb + 4 * lane] : 0u;
    }
    load(c, __shfl_sync(full, witem, pos));
    ++pos;
    return true;
  };
  // Each warp stages and reads only its own 64 columns, so the warps of a
  // CTA never wait for each other inside the loop.
  float4* const scw = sc + warp * 64;
  float* const suw = reinterpret_cast<float*>(su4 + warp * 16);
  auto stage = [&](const ColRegs& c, int slot) {
    stage_columns(scw + slot, column_in_frame<FORMULA>(c, ot));
    suw[slot + lane] = c.u;
  };
  ColRegs ca, cb;
  bool va = fetch(ca);
  bool vb = va && fetch(cb);
  while (va) {
    const unsigned ma = ca.m, mb = vb ? cb.m : 0u;
    __syncwarp();
    stage(ca, 0);
    if (vb) stage(cb, 32);
    __syncwarp();
    const bool na = vb && fetch(ca);
    const bool nbv = na && fetch(cb);
    if (a.prof_pairs)
      evaluated += 2 * SUBTILE * 32 * (((ma & 3u) != 0) + ((ma & 12u) != 0) +
                                       ((mb & 3u) != 0) + ((mb & 12u) != 0));
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    accumulate_item<FORMULA, F32_QU>(ma, scw, su4 + warp * 16, R, acc);
    if (EPI == EPI_MAP) {
      // the map keeps 32-term FP32 partials: each item is folded on its own
      kahan_add(s0, c0, acc[0]);
      kahan_add(s1, c1, acc[1]);
      kahan_add(s2, c2, acc[2]);
      kahan_add(s3, c3, acc[3]);
      acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
    }
    accumulate_item<FORMULA, F32_QU>(mb, scw + 32, su4 + warp * 16 + 8, R, acc);
    kahan_add(s0, c0, acc[0]);
    kahan_add(s1, c1, acc[1]);
    kahan_add(s2, c2, acc[2]);
    kahan_add(s3, c3, acc[3]);
    va = na;
    vb = nbv;
  }
  if (a.prof_pairs && lane == 0) atomicAdd(a.prof_pairs, (unsigned long long)evaluated);
  // Cross-warp reduction of the four column slices, in FP64.
  sred[warp][lane] = s0 - c0;
  sred[warp][lane + 32] = s1 - c1;
  sred[warp][lane + 64] = s2 - c2;
  sred[warp][lane + 96] = s3 - c3;
  __syncthreads();
  const double sum = ((double)sred[0][tid] + (double)sred[1][tid]) +
                     ((double)sred[2][tid] + (double)sred[3][tid]);
  const int i = base + tid;
  if (EPI == EPI_PRODUCT) {
    // q_i = wl_i var_s 2^-a_i sum_j e_ij wr_j v_j + e_i v_i
    const float q = fmaf(a.rowf[i], (float)sum, a.ediag[i] * a.vrow[i]);
    a.out[i] = q;
    if (DOT) {
      const double s = block_sum<TILE>((double)a.dotv[i] * (double)q, red);
      if (tid == 0) a.dot_partial[t] = s;
      if (last_block_arrive(a.counter)) {
        const double pq = reduce_partials<TILE>(a.dot_partial, gridDim.x, 1, 0, red);
        if (tid == 0) {
          *a.den_out = pq;
          *a.alpha_out = *a.num / pq;
          *a.counter = 0;
        }
      }
    }
  } else {
    // map: m_i = var_s * row factor * sum, accumulated in FP64
    const int dst = a.row_perm[i];
    if (dst >= 0) a.out64[dst] = (double)a.rowf[i] * sum;
  }
}

template <int FORMULA>
void launch_formula(int epi, const F32Args& a, cudaStream_t st) {
  const dim3 grid(a.n_row_tiles), block(TILE);
  if (epi == EPI_PRODUCT) {
    if (a.dot_partial)
      k_pair_f32<FORMULA, EPI_PRODUCT, true><<<grid, block, 0, st>>>(a);
    else
      k_pair_f32<FORMULA, EPI_PRODUCT, false><<<grid, block, 0, st>>>(a);
  } else if (epi == EPI_MAP) {
    k_pair_f32<FORMULA, EPI_MAP, false><<<grid, block, 0, st>>>(a);
  } else {
    throw Error{DS_ERR_ARG, "bad FP32 pair epilogue"};
  }
}

}  // namespace

void launch_pair_f32(int formula, int epi, const F32Args& a0, cudaStream_t st) {
  if (a0.n_row_tiles <= 0) return;
  F32Args a = a0;
  cudaEvent_t ev = nullptr;
  const int kind = epi == EPI_MAP ? 2 : 1;
  if (a.prof && a.prof->enabled) {
    a.prof_pairs = a.prof->d_pairs + kind;
    a.prof->begin(st, &ev);
  } else {
    a.prof_pairs = nullptr;
  }
  if (formula == F32_EXPANDED)
    launch_formula<F32_EXPANDED>(epi, a, st);
  else
    launch_formula<F32_DIRECT>(epi, a, st);
  DS_CHECK_LAUNCH();
  if (ev) a.prof->end(st, ev, kind);
}

}  // namespace ds
