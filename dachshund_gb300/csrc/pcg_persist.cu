// Small Jacobi-PCG solves (lib/pcg.h:27-160) from the stored pair values as one
// cooperative launch.
//
// Up to a few thousand pixels an iteration of the per-kernel form (pcg.cu) is
// all latency: three launches of a few microseconds each whose time goes into
// launch ramps, dependent loads and chains of dependent FP64 instructions
// (66 clocks each, 300 with 16 warps of an SM at them).  Here every 32-row slice of the value list has a
// CTA of its own for the whole solve: its values and columns stay in shared
// memory as far as they fit, its rows' x, r, d, s in one warp's registers, and
// an iteration is one gathered product and three grid barriers (q = A d and d.q;
// r.s and |r|^2; the new d's weights).  Same recurrence, same stopping rule, all
// FP64; every CTA forms the scalars from the same partials in the same order.
//
// Measured (4,096 pixels, table kernel, 203 iterations): 6.2 -> 4.3 ms; 7,100
// pixels, exact kernel: 366 -> 18.9 ms against evaluating the pairs.
//
// Barrier waits are bounded (SM clocks): a CTA that runs out sets the error word
// and leaves, the others find it and leave, and the call returns DS_ERR_TIMEOUT.
#include <algorithm>

#include "ds_device.cuh"
#include "ds_ops.h"

namespace ds {

namespace {

constexpr int NT = 512, W = NT / 32;

struct Args {
  int max_iter, step_r, cap;  // cap: entry rows kept in shared memory
  const int* cnt;
  const long long* start;
  const double* val;
  const double *wl, *wr, *e, *b, *pdiag;
  double var_s;
  double *x, *u, *ux;  // u, ux: column weights of d and of x
  double* part;        // 3 per CTA
  PcgState* st;
  double *hist, *dhist;
  unsigned int* bar;  // count, error
  long long limit;
};

struct Shared {
  double part[W][33];
  double row[32];
  int ok, done;
};

// Grid barrier in two halves, as persist.cu's (one monotonic count, added to
// with release and polled with acquire).
__device__ void grid_arrive(const Args& a) {
  __syncthreads();
  if (threadIdx.x == 0)
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
}

__device__ bool grid_wait(const Args& a, Shared& sm, unsigned int& epoch) {
  if (threadIdx.x == 0) {
    ++epoch;
    const unsigned int target = epoch * gridDim.x;
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

__device__ __forceinline__ bool grid_sync(const Args& a, Shared& sm, unsigned int& epoch) {
  grid_arrive(a);
  return grid_wait(a, sm, epoch);
}

// Sum over the warp, in every lane (the xor tree adds the same pairs everywhere).
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum of n partials (stride apart) by one warp, in every lane: two chains per
// lane, then the tree.
__device__ __forceinline__ double total(const double* part, int n, int stride) {
  double v0 = 0.0, v1 = 0.0;
  for (int i = threadIdx.x & 31; i < n; i += 64) {
    v0 += __ldcg(part + (size_t)i * stride);
    if (i + 32 < n) v1 += __ldcg(part + (size_t)(i + 32) * stride);
  }
  return warp_sum(v0 + v1);
}

template <class I>
__global__ void __launch_bounds__(NT) k_pcg_persistent(Args a, const I* __restrict__ cols) {
  extern __shared__ __align__(16) double vsm[];  // cap x 32 values, then columns
  __shared__ Shared sm;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int s = blockIdx.x, G = gridDim.x, i = s * 32 + lane;
  I* csm = reinterpret_cast<I*>(vsm + (size_t)a.cap * 32);
  const long long s0 = a.start[s];
  const int len = (int)(a.start[s + 1] - s0), n = a.cnt[i];
  const double* g = a.val + s0 * 32;
  const I* c = cols + s0 * 32;
  for (int k = tid; k < min(len, a.cap) * 32; k += NT) {
    vsm[k] = g[k];  // (padding entries too: never used)
    csm[k] = c[k];
  }
  __syncthreads();
  unsigned int epoch = 0;
  // Row sums of the slice's values with the weights u (written by every CTA
  // before a barrier), in warp 0's lanes: warp w takes entries w, w + 16, ..., in
  // two chains; two rows per warp add the 16 warps' sums by a tree.
  auto product = [&](const double* u) {
    double acc0 = 0.0, acc1 = 0.0;
    const int in = min(n, a.cap);
    int e = warp;
#pragma unroll 4
    for (; e + W < in; e += 2 * W) {
      const double u0 = __ldcg(u + csm[e * 32 + lane]), u1 = __ldcg(u + csm[(e + W) * 32 + lane]);
      acc0 = fma(vsm[e * 32 + lane], u0, acc0);
      acc1 = fma(vsm[(e + W) * 32 + lane], u1, acc1);
    }
#pragma unroll 4
    for (; e < n; e += W) {
      const size_t k = (size_t)e * 32 + lane;
      const bool here = e < in;
      const int j = here ? csm[k] : c[k];
      acc0 = fma(here ? vsm[k] : g[k], __ldcg(u + j), acc0);
    }
    sm.part[warp][lane] = acc0 + acc1;
    __syncthreads();
    double v = sm.part[lane & 15][2 * warp + (lane >> 4)];
    for (int o = 8; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o, 16);
    if ((lane & 15) == 0) sm.row[2 * warp + (lane >> 4)] = v;
    __syncthreads();
    return sm.row[lane];
  };
  // warp 0: the slice's rows
  const bool own = warp == 0;
  double wl = 0, wr = 0, ei = 0, b = 0, pd = 1, x = 0, r = 0, d = 0, sv = 0;
  double delta = 0, norm = 0;
  const double tol_norm_b = a.st->tol_norm_b;
  int it = 0, converged = 0;
  if (own) {
    wl = a.wl[i];
    wr = a.wr[i];
    ei = a.e[i];
    b = a.b[i];
    pd = a.pdiag[i];
    x = a.x[i];
    a.ux[i] = a.var_s * (wr * x);
  }
  // r = b - A x; d = M^-1 r; delta = r.d; |r|  (lib/pcg.h:95-108)
  if (!grid_sync(a, sm, epoch)) return;
  {
    const double q = product(a.ux);
    if (own) {
      r = b - (wl * q + ei * x);
      d = sv = r / pd;
      a.u[i] = a.var_s * (wr * d);
      const double rs = warp_sum(r * sv), rr = warp_sum(r * r);
      if (lane == 0) {
        a.part[G + 2 * s] = rs;
        a.part[G + 2 * s + 1] = rr;
      }
    }
  }
  if (!grid_sync(a, sm, epoch)) return;
  if (own) {
    delta = total(a.part + G, G, 2);
    norm = sqrt(total(a.part + G + 1, G, 2));
    if (s == 0 && lane == 0) {
      a.hist[0] = norm;
      a.dhist[0] = delta;
    }
  }
  for (it = 1; it < a.max_iter; ++it) {
    // q = A d, alpha = delta / d.q  (lib/pcg.h:34-39)
    const double acc = product(a.u);
    double q = 0.0;
    if (own) {
      q = wl * acc + ei * d;
      const double dq = warp_sum(d * q);
      if (lane == 0) a.part[s] = dq;
    }
    if (!grid_sync(a, sm, epoch)) return;
    const bool full = it % a.step_r == 0;
    if (own) {
      const double alpha = delta / total(a.part, G, 1);
      x = fma(alpha, d, x);
      r = fma(-alpha, q, r);
      if (full) a.ux[i] = a.var_s * (wr * x);
    }
    if (full) {  // r = b - A x
      if (!grid_sync(a, sm, epoch)) return;
      const double ax = product(a.ux);
      if (own) r = b - (wl * ax + ei * x);
    }
    if (own) {
      sv = r / pd;  // lib/pcg.h:52
      const double rs = warp_sum(r * sv), rr = warp_sum(r * r);
      if (lane == 0) {
        a.part[G + 2 * s] = rs;
        a.part[G + 2 * s + 1] = rr;
      }
    }
    if (!grid_sync(a, sm, epoch)) return;
    if (own) {
      const double rs = total(a.part + G, G, 2);
      const double beta = rs / delta;  // lib/pcg.h:58-61
      delta = rs;
      d = fma(beta, d, sv);
      a.u[i] = a.var_s * (wr * d);
    }
    grid_arrive(a);
    if (own) {  // while the barrier completes
      norm = sqrt(total(a.part + G + 1, G, 2));
      if (s == 0 && lane == 0) {
        a.hist[it] = norm;
        a.dhist[it] = delta;
      }
      if (lane == 0) sm.done = norm <= tol_norm_b;  // lib/pcg.h:130
    }
    if (!grid_wait(a, sm, epoch)) return;  // the new weights; sm.done
    if (sm.done) {
      converged = 1;
      ++it;
      break;
    }
  }
  if (own) a.x[i] = x;
  if (s == 0 && tid == 0) {
    a.st->iter = it - 1;
    a.st->norm_r = norm;
    a.st->delta = delta;
    a.st->done = 1;
    a.st->converged = converged;
  }
}

}  // namespace

// The whole iteration of run_pcg (x, the state's norm and tolerance set) when
// every slice gets a resident CTA, two to an SM at most (n up to 9,728 on 152
// SMs); false leaves it to the per-kernel form, which at larger n spends its time
// in the product and not between kernels.  Launches only: the caller reads the error
// word pcg_sync[1] once the stream has finished.
bool run_pcg_persistent(ds_operator* op, const ds_pcg_params& pp, cudaStream_t st) {
  const PairVals& pv = op->vals;
  const int ns = op->pix.n_pad / 32, sms = op->ctx->num_sms;
  if (ns > 2 * sms || pp.max_iter < 2) return false;
  const bool narrow = pv.col16.p != nullptr;
  const void* fn = narrow ? (const void*)k_pcg_persistent<unsigned short>
                          : (const void*)k_pcg_persistent<int>;
  // shared memory of one CTA per SM, or of two
  const size_t bytes = ns <= sms ? 200 * 1024 : 96 * 1024;
  if ((long long)resident_ctas(fn, NT, bytes) * sms < ns) return false;
  op->ud.alloc(op->pix.n_pad);
  op->u.alloc(op->pix.n_pad);
  op->pcg_sync.alloc(2);
  DS_CUDA(cudaMemsetAsync(op->pcg_sync.p, 0, op->pcg_sync.bytes(), st));
  Args a{};
  a.max_iter = pp.max_iter;
  a.step_r = pp.step_r;
  a.cap = (int)(bytes / (32 * (sizeof(double) + (narrow ? 2 : 4))));
  a.cnt = pv.cnt.p;
  a.start = pv.start.p;
  a.val = pv.val.p;
  a.wl = op->wl.p;
  a.wr = op->wr.p;
  a.e = op->e.p;
  a.b = op->b.p;
  a.pdiag = op->pdiag.p;
  a.var_s = op->kc.var_s;
  a.x = op->x.p;
  a.u = op->ud.p;
  a.ux = op->u.p;
  a.part = op->partial2.p;  // at least 2,048 + 2 n_pad
  a.st = op->state.p;
  a.hist = op->hist.p;
  a.dhist = op->dhist.p;
  a.bar = op->pcg_sync.p;
  a.limit = op->ctx->wait_limit > 0 ? op->ctx->wait_limit : 4000000000LL;
  const unsigned short* c16 = pv.col16.p;
  const int* c32 = pv.col32.p;
  void* args[] = {&a, narrow ? (void*)&c16 : (void*)&c32};
  launch_cooperative(fn, ns, NT, args, bytes, st);
  return true;
}

}  // namespace ds
