// Persistent form of the mixed-precision iteration for pixels on no common grid:
// Jacobi-PCG with the FP32 pair kernels' product (pair_f32.cu), one cooperative
// launch of all iterations up to the next reliable update.
//
// The per-kernel form (mixed.cu) takes one CTA per 128-row tile: too few warps in
// flight (9 per SM at 44,237 pixels, none on half the SMs below 10,000), tiles of
// uneven weight, and a chain of five dependent loads before each launch's first
// exponential.  The product's unit here is a round: 64 columns against the 128 rows
// of a tile, one FP32 sum per row.  All rounds of all tiles are shared out evenly
// over all warps, whose round list and row data stay in registers from one
// iteration to the next; a round's 128 sums go to a buffer in L2, and the row's
// owner folds them into the compensated sums of the tile's four slices in the
// per-kernel form's order: every FP32 value is that form's bit for bit.
//
// Phases, a grid barrier after each: the rounds (p = z + beta p formed as the
// columns are loaded); the rows' q and p.q; r, z (then x) and the sums r.z, |r|^2.
// Rows are owned by thread, and the FP64 sums are the per-kernel form's to the last
// bit, order included: a Krylov recurrence in FP32 amplifies any flipped rounding to
// a few percent of the final residual, which an FP32 evaluation of the map from x
// shows.  A dependent FP64 addition takes 66 clocks with up to 4 warps of an SM at
// it but 300 with 16, so one warp adds up what the shuffles of 4 or 8 would (tree).
//
// Measured (solve and map on a kept operator, per-kernel form -> here): 2,048 pixels
// 5.0 -> 3.1 ms, 10,240 7.4 -> 4.2, 24,000 8.9 -> 5.9, 44,237 12.2 -> 9.0.  An
// iteration of 44,237 pixels takes 68,000 clocks: 36,000 the rounds (18,000 if the
// exponentials alone bound them), 9,000 their uneven ends and barrier, 11,000 the rows,
// 12,000 the step and its sums.
#include <algorithm>
#include <string>

#include <cub/device/device_scan.cuh>

#include "ds_device.cuh"
#include "ds_f32.h"
#include "ds_ff.cuh"
#include "ds_mixed_dev.cuh"
#include "ds_ops.h"
#include "ds_pair_f32.cuh"

namespace ds {

namespace {

constexpr int NT = 512, W = NT / 32, QUADS = NT / TILE;
constexpr int VB = 256;     // rows per block of the vector sums
// Rows per thread at most: 155,648 pixels.  131,072 pixels take 26.4 ms per solve in
// the per-kernel form and 22.6 here; 262,144 take 44.4 and 45.8 (the tiles then fill
// the SMs evenly without it, and the rounds' sums leave L2).
constexpr int MAX_PER = 2;

// A thread's row (registers are the rounds'); `per` of them per thread.
struct Row {
  double x;
  float p, r, z, q, pd, rowf, ed, pad;
};

struct Args {
  int n_tiles, max_iter, per, g;
  const int4* rounds;         // tile, item, item or 0, -
  const int* round_ptr;       // first round of (tile, slice); 4 n_tiles + 1
  const int* warp_ptr;        // first round of a warp; W G + 1
  const float4* xi;           // tile-relative coordinates, colw
  const float4* orig;
  const float *rowf, *ediag, *pd;
  double* x;
  float *p, *r, *z;
  float2* zp;                 // (z, p) of every pixel
  float4* sums;               // rounds x 32: lane l's rows l, l + 32, l + 64, l + 96
  double* part;               // p.q per tile, then r.z and |r|^2 per row block
  MixedState* st;
  double* hist;
  unsigned int* bar;          // arrivals, error
  long long limit;
};

struct Shared {
  float4 sc[W * 64];   // per warp: 64 staged columns
  float4 su4[W * 16];  // and their values
  double sum[2][NT];   // sums in progress (r.z and |r|^2)
  MixedState s;
  float slice[QUADS][4][TILE];
  int ok;
};

// The sum that NW warps' block_sum would form of v[0 .. 32 NW), by one warp (valid in
// lane 0; v is overwritten).
template <int NW>
__device__ __forceinline__ double tree(double* v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
#pragma unroll
    for (int e = lane; e < NW * s; e += 32) {
      const int i = (e / s) * 32 + e % s;
      v[i] += v[i + s];
    }
    __syncwarp();
  }
  double t = 0.0;
  if (lane == 0)
#pragma unroll
    for (int w = 0; w < NW; ++w) t += v[32 * w];
  return t;
}

// float(((s0 + s1) + s2 + s3) in FP64) of the slices' sums: in FP32 with the exact
// errors, in FP64 where these leave the rounding open (one row in millions).
__device__ __forceinline__ float slice_total(float s0, float s1, float s2, float s3) {
  float a, ea, b, eb, s, es;
  two_sum(s0, s1, a, ea);
  two_sum(s2, s3, b, eb);
  two_sum(a, b, s, es);
  const float rest = __fadd_rn(__fadd_rn(ea, eb), es);
  const float open = 4e-7f * (fabsf(ea) + fabsf(eb) + fabsf(es));
  const float lo = __fadd_rn(s, __fadd_rn(rest, -open)), hi = __fadd_rn(s, __fadd_rn(rest, open));
  if (lo == hi) return lo;
  return (float)(((double)s0 + (double)s1) + ((double)s2 + (double)s3));
}

__device__ __forceinline__ void grid_arrive(const Args& a) {
  __syncthreads();
  if (threadIdx.x == 0)
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
}

__device__ __forceinline__ bool grid_wait(const Args& a, Shared& sm, unsigned int& epoch) {
  if (threadIdx.x == 0) {
    const unsigned int target = ++epoch * gridDim.x;
    const long long t0 = clock64();
    int ok = 1;
    for (int k = 0;; ++k) {
      if (clock64() - t0 >= a.limit) {
        atomicExch(a.bar + 1, epoch);
        ok = 0;
        break;
      }
      unsigned int f;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(a.bar) : "memory");
      if ((int)(f - target) >= 0) break;
      if ((k & 15) == 15 && *(volatile unsigned int*)(a.bar + 1)) {
        ok = 0;
        break;
      }
    }
    sm.ok = ok;
  }
  __syncthreads();
  return sm.ok != 0;
}

template <int FORMULA>
__global__ void __launch_bounds__(NT, 1) k_mixed_pairs(Args a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  Shared& sm = *reinterpret_cast<Shared*>(smraw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, G = gridDim.x;
  constexpr unsigned full = 0xffffffffu;
  if (tid == 0) sm.s = *a.st;
  // Half a CTA owns the rows of block vb of the vector sums, rows vb VB + ... and
  // every g VB rows on; a quad of warps a tile of them.
  const int quad = tid / TILE, row = tid % TILE, slice = row >> 5;
  const int vb = (int)blockIdx.x + G * (tid / VB);
  Row* const rows = reinterpret_cast<Row*>(smraw + sizeof(Shared)) + tid;  // k-th at k NT
  auto tile_of = [&](int k) {
    return vb < a.g ? 2 * (vb + k * a.g) + (quad & 1) : a.n_tiles;
  };
  for (int k = 0; k < a.per; ++k) {
    const int t = tile_of(k);
    if (t >= a.n_tiles) break;
    const int g = t * TILE + row;
    Row w;
    w.x = a.x[g];
    w.p = a.p[g];
    w.r = a.r[g];
    w.z = a.z[g];
    w.q = w.pad = 0.f;
    w.pd = a.pd[g];
    w.rowf = a.rowf[g];
    w.ed = a.ediag[g];
    rows[k * NT] = w;
    a.zp[g] = make_float2(w.z, w.p);
  }
  // the warp's rounds: consecutive ones, neighbouring ranges on different SMs
  const int gw = warp * G + (int)blockIdx.x;
  const int r0 = a.warp_ptr[gw], nr = a.warp_ptr[gw + 1] - r0;
  int4 ent = make_int4(0, 0, 0, 0);  // lane l: round l of the batch
  if (lane < nr) ent = a.rounds[r0 + lane];
  int cur = -1;  // the tile whose rows are held
  RowRegs R{};
  float4 ot = make_float4(0.f, 0.f, 0.f, 0.f);
  float4* const scw = sm.sc + warp * 64;
  float* const suw = reinterpret_cast<float*>(sm.su4 + warp * 16);

  struct Col {
    float4 q;
    float4 o;
    float2 zp;
  };
  auto load = [&](Col& c, unsigned it) {
    const int ct = (int)(it >> 6);
    const int j = ct * TILE + 32 * (int)((it >> 4) & 3u) + lane;
    c.o = a.orig[ct];
    c.q = a.xi[j];
    c.zp = __ldcg(a.zp + j);
  };
  auto stage = [&](const Col& c, int slot, float beta) {
    ColRegs g;
    g.q = make_float3(c.q.x, c.q.y, c.q.z);
    g.o = make_float3(c.o.x, c.o.y, c.o.z);
    stage_columns(scw + slot, column_in_frame<FORMULA>(g, ot));
    suw[slot + lane] = c.q.w * fmaf(beta, c.zp.y, c.zp.x);
  };
  unsigned int epoch = 0;
  grid_arrive(a);
  if (!grid_wait(a, sm, epoch)) return;
  while (!sm.s.need_update && !sm.s.done && sm.s.iter < a.max_iter) {
    const int it = sm.s.iter + 1;
    const float beta = (float)sm.s.beta;
    // ---- the rounds
    if (nr > 0) {
      Col ca, cb;
      if (nr > 32) ent = a.rounds[r0 + lane];
      int t = __shfl_sync(full, ent.x, 0);
      unsigned ia = (unsigned)__shfl_sync(full, ent.y, 0);
      unsigned ib = (unsigned)__shfl_sync(full, ent.z, 0);
      load(ca, ia);
      load(cb, ib);
      for (int k = 0; k < nr; ++k) {
        if (t != cur) {
          cur = t;
          const float4* xr = a.xi + (size_t)t * TILE + lane;
#pragma unroll
          for (int c = 0; c < 4; ++c) R.set(c, xr[32 * c]);
          ot = a.orig[t];
        }
        const unsigned masks = (ia & 15u) | (ib & 15u) << 4;
        __syncwarp();
        stage(ca, 0, beta);
        stage(cb, 32, beta);
        __syncwarp();
        if (k + 1 < nr) {
          const int b = (k + 1) & 31;
          if (b == 0) ent = k + 1 + lane < nr ? a.rounds[r0 + k + 1 + lane] : ent;
          t = __shfl_sync(full, ent.x, b);
          ia = (unsigned)__shfl_sync(full, ent.y, b);
          ib = (unsigned)__shfl_sync(full, ent.z, b);
          load(ca, ia);
          load(cb, ib);
        }
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
        for (int h = 0; h < 2; ++h)
          accumulate_item<FORMULA, 8>((masks >> (4 * h)) & 15u, scw + 32 * h,
                                      sm.su4 + warp * 16 + 8 * h, R, acc);
        a.sums[(size_t)(r0 + k) * 32 + lane] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      }
    }
    grid_arrive(a);
    if (!grid_wait(a, sm, epoch)) return;
    // ---- the rows: q = A32 p and p.q
    for (int k = 0; k < a.per; ++k) {
      const int t = tile_of(k);
      const bool own = t < a.n_tiles;
      float(&sl)[4][TILE] = sm.slice[quad];
      if (own) {
        const int f0 = a.round_ptr[4 * t + slice], f1 = a.round_ptr[4 * t + slice + 1];
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
        float c0 = 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f;
        constexpr int U = 8;
        for (int f = f0; f < f1; f += U) {
          float4 v[U];
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (f + u < f1) v[u] = __ldcg(a.sums + (size_t)(f + u) * 32 + lane);
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (f + u < f1) {
              kahan_add(s0, c0, v[u].x);
              kahan_add(s1, c1, v[u].y);
              kahan_add(s2, c2, v[u].z);
              kahan_add(s3, c3, v[u].w);
            }
        }
        sl[slice][lane] = s0 - c0;
        sl[slice][lane + 32] = s1 - c1;
        sl[slice][lane + 64] = s2 - c2;
        sl[slice][lane + 96] = s3 - c3;
      }
      __syncthreads();
      if (own) {
        Row& w = rows[k * NT];
        const float p = fmaf(beta, w.p, w.z);
        const float sum = slice_total(sl[0][row], sl[1][row], sl[2][row], sl[3][row]);
        const float q = fmaf(w.rowf, sum, w.ed * p);
        w.p = p;
        w.q = q;
        sm.sum[0][tid] = (double)p * (double)q;
      }
      __syncthreads();
      if (own && slice == 0) {
        const double d = tree<TILE / 32>(sm.sum[0] + tid - lane);
        if (lane == 0) a.part[t] = d;
      }
    }
    grid_arrive(a);
    if (!grid_wait(a, sm, epoch)) return;
    // ---- the step
    if (warp < TILE / 32) {
      double v = 0.0;
      for (int k = tid; k < a.n_tiles; k += TILE) v += __ldcg(a.part + k);
      sm.sum[0][tid] = v;
    }
    __syncthreads();
    if (warp == 0) {
      const double pq = tree<TILE / 32>(sm.sum[0]);
      if (lane == 0) {
        sm.s.pq = pq;
        sm.s.alpha = sm.s.rz / pq;
      }
    }
    __syncthreads();
    const double alpha_d = sm.s.alpha;
    const float alpha = (float)alpha_d;
    {
      double rz = 0.0, rr = 0.0;
      for (int k = 0; k < a.per && tile_of(k) < a.n_tiles; ++k) {
        Row& w = rows[k * NT];
        const float r = fmaf(-alpha, w.q, w.r), z = r / w.pd;
        a.zp[tile_of(k) * TILE + row] = make_float2(z, w.p);
        w.r = r;
        w.z = z;
        rz = fma((double)r, (double)z, rz);
        rr = fma((double)r, (double)r, rr);
      }
      sm.sum[0][tid] = rz;
      sm.sum[1][tid] = rr;
    }
    __syncthreads();
    if ((warp & 3) == 0) {  // warps 0, 4: r.z, |r|^2 of the first half; 8, 12: the second
      const int h = (warp >> 2) & 1;
      const double d = tree<VB / 32>(sm.sum[h] + (warp >> 3) * VB);
      const int b = (int)blockIdx.x + G * (warp >> 3);
      if (lane == 0 && b < a.g) a.part[a.n_tiles + 2 * b + h] = d;
    }
    grid_arrive(a);
    for (int k = 0; k < a.per && tile_of(k) < a.n_tiles; ++k) {
      Row& w = rows[k * NT];
      w.x = fma(alpha_d, (double)w.p, w.x);
    }
    if (!grid_wait(a, sm, epoch)) return;
    {
      const int h = tid / VB;  // r.z by the first half of the CTA, |r|^2 by the second
      double v = 0.0;
      for (int k = tid % VB; k < a.g; k += VB) v += __ldcg(a.part + a.n_tiles + 2 * k + h);
      sm.sum[h][tid % VB] = v;
    }
    __syncthreads();
    if (warp == 0) {
      const double trz = tree<VB / 32>(sm.sum[0]);
      if (lane == 0) {
        sm.s.rz_old = sm.s.rz;
        sm.s.rz = trz;
        sm.s.beta = trz / sm.s.rz_old;
      }
    } else if (warp == VB / 32) {
      const double trr = tree<VB / 32>(sm.sum[1]);
      if (lane == 0) {
        sm.s.rnorm = sqrt(trr);
        sm.s.iter = it;
        if (blockIdx.x == 0) a.hist[it] = sm.s.rnorm;
        sm.s.rmax = fmax(sm.s.rmax, sm.s.rnorm);
        sm.s.need_update = update_due(&sm.s, it) ? 1 : 0;
        sm.s.skip_update = !sm.s.need_update;
      }
    }
    __syncthreads();
  }
  for (int k = 0; k < a.per && tile_of(k) < a.n_tiles; ++k) {
    const int g = tile_of(k) * TILE + row;
    const Row w = rows[k * NT];
    a.x[g] = w.x;
    a.p[g] = w.p;
    a.r[g] = w.r;
    a.z[g] = w.z;
  }
  if (blockIdx.x == 0 && tid == 0) {
    *a.st = sm.s;
  }
}

// Rounds of (tile, slice) i: two of the slice's items each.
__global__ void k_round_count(int n, const int* __restrict__ item_ptr, int* __restrict__ cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  int c = 0;
  if (i < n) {
    const int items = item_ptr[(i >> 2) + 1] - item_ptr[i >> 2];
    c = (((items - (i & 3) + 3) >> 2) + 1) >> 1;
  }
  cnt[i] = c;
}

// Time of an item's 32 columns: by the row pairs evaluated, and its loads.
__device__ __forceinline__ int item_weight(unsigned m) {
  return (m & 15u) ? 1 + 4 * (((m & 3u) != 0) + ((m & 12u) != 0)) : 0;
}

__global__ void k_round_fill(int n, const int* __restrict__ item_ptr,
                             const unsigned* __restrict__ items, const int* __restrict__ ptr,
                             int4* __restrict__ rounds, int* __restrict__ weight) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int t = i >> 2, i1 = item_ptr[t + 1];
  int k = item_ptr[t] + (i & 3);
  for (int r = ptr[i]; r < ptr[i + 1]; ++r, k += 8) {
    const unsigned a = items[k], b = k + 4 < i1 ? items[k + 4] : 0u;
    rounds[r] = make_int4(t, (int)a, (int)b, 0);
    weight[r] = 1 + item_weight(a) + item_weight(b);
  }
}

// The warps' shares: equal weights (`before` = the weight before each round).
__global__ void k_warp_rounds(int n_warps, int n_rounds, const int* __restrict__ before,
                              int* __restrict__ warp_ptr) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w > n_warps) return;
  const long long want = (long long)before[n_rounds] * w / n_warps;
  int lo = 0, hi = n_rounds;
  while (lo < hi) {
    const int m = (lo + hi) >> 1;
    if (before[m] < want)
      lo = m + 1;
    else
      hi = m;
  }
  warp_ptr[w] = lo;
}

__global__ void k_pack_xi(int n, const float4* __restrict__ xi, const float* __restrict__ colw,
                          float4* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = make_float4(xi[i].x, xi[i].y, xi[i].z, colw[i]);
}

}  // namespace

static const void* kernel_of(const OpF32& f) {
  return f.formula == F32_EXPANDED ? (const void*)k_mixed_pairs<F32_EXPANDED>
                                   : (const void*)k_mixed_pairs<F32_DIRECT>;
}

static void drop_rounds(OpF32& f) {
  f.rounds_built = false;
  for (auto* b : {&f.round_ptr, &f.warp_ptr}) b->release();
  f.rounds.release();
  f.round_sums.release();
  f.xiw.release();
  f.zp.release();
  f.round_part.release();
  f.round_bar.release();
}

static bool build_rounds(ds_operator* op, OpF32& f);

// Prepares the launches (kept with the operator's FP32 pair list); false when the
// rows do not fit or the rounds (536 bytes each; clumped pixels have millions) would
// take more than the context's share of the device memory, and the per-kernel form
// runs.  Decided again when the share is set; share 0 gives them back.
bool mixed_pairs_usable(ds_operator* op, OpF32& f, int g) {
  const int G = op->ctx->num_sms;
  const int per = (op->pix.n_pad + g * VB - 1) / (g * VB);
  if (per > MAX_PER || g > 2 * G) return false;
  const size_t smem = sizeof(Shared) + (size_t)per * NT * sizeof(Row);
  const void* fn = kernel_of(f);
  if (resident_ctas(fn, NT, smem) < 1) return false;
  if (f.rounds_decided == op->ctx->share_serial) return f.rounds_built;
  if (!(f.rounds_built && op->ctx->store_share > 0.0)) {
    drop_rounds(f);
    try {
      f.rounds_built = op->ctx->store_share > 0.0 && build_rounds(op, f);
    } catch (const Error& e) {
      drop_rounds(f);
      if (e.code != DS_ERR_OOM) throw;
      cudaGetLastError();  // the failed allocation's
    }
    if (!f.rounds_built) drop_rounds(f);
  }
  f.rounds_decided = op->ctx->share_serial;
  return f.rounds_built;
}

// The rounds, their shares and the buffers; false when over the budget.
static bool build_rounds(ds_operator* op, OpF32& f) {
  const int nt = op->pix.n_tiles, G = op->ctx->num_sms;
  cudaStream_t st = op->ctx->stream;
  const int n = 4 * nt, nw = W * G;
  DevBuf<int> cnt, before;
  DevBuf<unsigned char> tmp;
  auto scan = [&](const int* in, int* out, int m) {
    size_t bytes = 0;
    DS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, m, st));
    tmp.alloc(std::max<size_t>(bytes, 1));
    DS_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, bytes, in, out, m, st));
  };
  cnt.alloc(n + 1);
  f.round_ptr.alloc(n + 1);
  k_round_count<<<n / 256 + 1, 256, 0, st>>>(n, f.pairs.item_ptr.p, cnt.p);
  DS_CHECK_LAUNCH();
  scan(cnt.p, f.round_ptr.p, n + 1);
  int total = 0;
  DS_CUDA(cudaMemcpyAsync(&total, f.round_ptr.p + n, sizeof(int), cudaMemcpyDeviceToHost, st));
  DS_CUDA(cudaStreamSynchronize(st));
  if ((size_t)total * (32 * sizeof(float4) + sizeof(int4) + 2 * sizeof(int)) >
      store_budget(op->ctx))
    return false;
  f.rounds.alloc(std::max(total, 1));
  DevBuf<int> weight;
  weight.alloc(total + 1);
  before.alloc(total + 1);
  DS_CUDA(cudaMemsetAsync(weight.p + total, 0, sizeof(int), st));
  k_round_fill<<<n / 256 + 1, 256, 0, st>>>(n, f.pairs.item_ptr.p, f.pairs.items.p,
                                            f.round_ptr.p, f.rounds.p, weight.p);
  DS_CHECK_LAUNCH();
  scan(weight.p, before.p, total + 1);
  f.warp_ptr.alloc(nw + 1);
  k_warp_rounds<<<nw / 256 + 1, 256, 0, st>>>(nw, total, before.p, f.warp_ptr.p);
  DS_CHECK_LAUNCH();
  f.round_sums.alloc((size_t)std::max(total, 1) * 32);
  f.xiw.alloc(op->pix.n_pad);
  k_pack_xi<<<op->pix.n_pad / 256 + 1, 256, 0, st>>>(op->pix.n_pad, f.pts.xi.p, f.colw.p,
                                                     f.xiw.p);
  DS_CHECK_LAUNCH();
  f.zp.alloc(op->pix.n_pad);
  f.round_part.alloc((size_t)nt + 4 * G);
  f.round_bar.alloc(2);
  return true;
}

// Iterations up to the next reliable update (or the cap) from x, p, r, z and the
// state.
void launch_mixed_pairs(ds_operator* op, OpF32& f, double* X, int max_iter, int g,
                        cudaStream_t st) {
  DS_CUDA(cudaMemsetAsync(f.round_bar.p, 0, f.round_bar.bytes(), st));
  const int G = op->ctx->num_sms;
  Args a{};
  a.n_tiles = op->pix.n_tiles;
  a.max_iter = max_iter;
  a.g = g;
  a.per = (op->pix.n_pad + g * VB - 1) / (g * VB);
  a.rounds = f.rounds.p;
  a.round_ptr = f.round_ptr.p;
  a.warp_ptr = f.warp_ptr.p;
  a.xi = f.xiw.p;
  a.orig = f.pts.orig.p;
  a.rowf = f.rowf.p;
  a.ediag = f.ediag.p;
  a.pd = f.pdiag.p;
  a.x = X;
  a.p = f.p.p;
  a.r = f.r.p;
  a.z = f.z.p;
  a.zp = f.zp.p;
  a.sums = f.round_sums.p;
  a.part = f.round_part.p;
  a.st = f.state.p;
  a.hist = f.hist.p;
  a.bar = f.round_bar.p;
  a.limit = op->ctx->wait_limit > 0 ? op->ctx->wait_limit : 4000000000LL;
  void* args[] = {&a};
  launch_cooperative(kernel_of(f), G, NT, args, sizeof(Shared) + (size_t)a.per * NT * sizeof(Row),
                     st);
}

}  // namespace ds
