// The learned preconditioner's message-passing layers at inference, on the
// tensor cores: out = h + relu(Z), Z = [h | A_z h | A_n h] W + b, with h the
// activations [M x 128] (FP32, row-major), W [384 x 128] (the BF16 forward
// weights, exact in TF32) and M a multiple of 128.  tcgen05.mma kind::tf32
// (M = N = 128, K = 8): the activations enter as TF32 (10-bit mantissa), a
// relative perturbation near 1e-3 of the hidden state against the FP32
// CUDA-core GEMM that training uses (whose gradients the CPU oracle checks);
// the preconditioner built from it differs correspondingly little, and the
// solve it preconditions still stops on its FP64-accurate residual.
//
// The aggregated activations [M x 384] are never stored: the kernel's producer
// warps form them from h (11 rows of h per row, mostly L2 hits) straight into
// the MMA's operand layout, with the sums of k_agg_fwd in its order.  Writing
// and reading them back cost 0.8 GB of HBM traffic per layer; W^T staged by the
// same threads cost as many shared-memory stores as the activations, and comes
// by bulk copies instead.  Bound now by the producers' L2 reads (0.72 MB per
// 128-row tile, 7 TB/s).  Measured at 262,144 rows: 210 us per layer, 472 us
// with the aggregation as a kernel of its own; the same bits.
//
// Per CTA (one per SM, persistent over 128-row tiles):
//   * warps 0-15 form K chunks of 32 of the tile's 128 rows (chunks 0-3 h, 4-7
//     A_z h, 8-11 A_n h) in 4 shared-memory stages, in the canonical K-major
//     no-swizzle layout: 4 rows by 32 channels per warp access (whole 128-byte
//     lines: 4 L1 wavefronts each, where 8 rows by 64 bytes took 32 and the L1
//     wavefronts bound the kernel), conflict-free shared stores; thread 0 also starts the bulk copy of the chunk's W^T
//     (16 KB, stored in the operand layout by k_wt_f32);
//   * lane 0 of warp 20 issues 4 MMAs per chunk into one of two TMEM
//     accumulators (128 columns each) and commits them;
//   * warps 16-19 read an accumulator back (warp w: TMEM lanes 32 (w % 4) ..,
//     its rows), add the bias, apply relu and the residual and store out,
//     overlapping the next tile's MMAs.
// Every mbarrier wait is bounded (error code, then a clean exit).
#include "ds_device.cuh"
#include "ds_learned.h"
#include "ds_tc.cuh"

#include <cuda_bf16.h>

#include <algorithm>

namespace ds {
namespace {

constexpr int LG_K = 384;            // 3 H
constexpr int LG_N = 128;            // H
constexpr int LG_KC = 32;            // K per stage
constexpr int LG_NCH = LG_K / LG_KC;
constexpr int LG_STAGES = 4;
constexpr int LG_PW = 16;             // producer warps
constexpr int LG_PR = 128 / LG_PW;    // rows of a tile per producer warp
constexpr int LG_PJ = LG_PR / 4;      // rows per lane
constexpr int LG_THREADS = (LG_PW + 5) * 32;
constexpr int LG_OPF = 128 * LG_KC;  // floats of one 128-row operand chunk (16 KB)
constexpr uint32_t LG_LBO = 16 * 128;
constexpr uint32_t LG_SBO = 128;
constexpr uint32_t LG_IDESC = idesc_tf32(128, LG_N);

// The A operand's core-matrix columns lie 16 bytes further apart than packed, so
// that 8 lanes storing 8 consecutive 4-channel groups of one row hit 8 different
// bank groups.
constexpr uint32_t LG_LBO_A = LG_LBO + 16;
constexpr int LG_OPF_A = LG_KC / 4 * (int)LG_LBO_A / 4;
constexpr int LG_TW = 36;            // floats per row of the epilogue's transpose

struct LgSmem {
  float a[LG_STAGES][LG_OPF_A];
  float b[LG_STAGES][LG_OPF];
  float t[4][32][LG_TW];
  int nb[128][8];                    // the tile rows' neighbours: row of h
  float g[128][8];                   // and weight
  uint64_t full[LG_STAGES], empty[LG_STAGES], b_full[LG_STAGES];
  uint64_t d_full[2], d_empty[2];
  uint32_t tmem_addr;
  int abort;
};
constexpr size_t LG_SMEM_BYTES = sizeof(LgSmem) + 1024;

// element (row r, k) of a 128-row chunk with K = 32 (8 core-matrix columns)
__device__ __forceinline__ int lg_at(int r, int k) {
  return ((k >> 2) * 16 + (r >> 3)) * 32 + (r & 7) * 4 + (k & 3);
}

__device__ __forceinline__ int lg_at_a(int r, int k) {
  return (k >> 2) * ((int)LG_LBO_A / 4) + (r >> 3) * 32 + (r & 7) * 4 + (k & 3);
}

__device__ __forceinline__ bool lg_wait(LgSmem& sm, uint64_t* bar, uint32_t parity, int* err,
                                        int code) {
  if (mbar_wait(bar, parity)) return true;
  atomicExch(err, code);
  *(volatile int*)&sm.abort = 1;
  return false;
}

__device__ __forceinline__ bool lg_warp_wait(LgSmem& sm, uint64_t* bar, uint32_t parity,
                                             int* err, int code, int lane) {
  int ok = 1;
  if (lane == 0) ok = lg_wait(sm, bar, parity, err, code);
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();
  return ok != 0;
}

// W^T as FP32 from the BF16 forward weights [384 x 128], in the operand layout,
// chunk after chunk of 32 k.
__global__ void k_wt_f32(const __nv_bfloat16* __restrict__ w, float* __restrict__ wt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= LG_K * LG_N) return;
  const int k = i / LG_N, n = i % LG_N;
  wt[(size_t)(k / LG_KC) * LG_OPF + lg_at(n, k % LG_KC)] = __bfloat162float(w[i]);
}

__device__ __forceinline__ float4 f4_add(float4 a, float4 b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

__device__ __forceinline__ float4 f4_fma(float g, float4 v, float4 a) {
  return make_float4(fmaf(g, v.x, a.x), fmaf(g, v.y, a.y), fmaf(g, v.z, a.z), fmaf(g, v.w, a.w));
}

// Tile t of the launch order: with whole tiles per skewer, the first tile of
// every skewer, then the second, ..., so that the rows in use (every skewer's
// neighbours at one z range) stay in L2.
__device__ __forceinline__ int lg_tile(int t, int n_tiles, int n_per) {
  if (n_per % 128) return t;
  const int per = n_per / 128, n_sk = n_tiles / per;
  return t % n_sk * per + t / n_sk;
}

__global__ void __launch_bounds__(LG_THREADS, 1)
    k_layer_tc(int M, int n_per, const float* __restrict__ h, const int* __restrict__ nbr,
               const float* __restrict__ gw, const float* __restrict__ wt,
               const float* __restrict__ bias, float* __restrict__ out, int* err) {
  extern __shared__ uint8_t lg_raw[];
  LgSmem& sm = *reinterpret_cast<LgSmem*>((reinterpret_cast<uintptr_t>(lg_raw) + 1023) &
                                          ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < LG_STAGES; ++s) {
      mbar_init(&sm.full[s], LG_PW);
      mbar_init(&sm.empty[s], 1);
      mbar_init(&sm.b_full[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.d_full[b], 1);
      mbar_init(&sm.d_empty[b], 4);
    }
    sm.abort = 0;
    mbar_fence_init();
  }
  if (warp == 0) tmem_alloc(&sm.tmem_addr, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_addr;
  const int n_tiles = M / 128;
  int last = -1;

  if (warp < LG_PW) {
    // ---- producers: lane (rr, c4) = (lane / 8, lane % 8) holds rows LG_PR
    // warp + 4 j + rr, channels 4 c4 .. of the chunk's 32
    const int rr = lane >> 3, c4 = lane & 7;
    uint32_t g = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
      const int tile = lg_tile(t, n_tiles, n_per);
      const int row0 = tile * 128 + LG_PR * warp;
      __syncwarp();  // the previous tile's table is read
      for (int q = lane; q < LG_PR * 8; q += 32) {
        const int i = row0 + (q >> 3), s = i / n_per, m = q & 7;
        sm.nb[LG_PR * warp + (q >> 3)][m] = nbr[s * 8 + m] * n_per + (i - s * n_per);
        sm.g[LG_PR * warp + (q >> 3)][m] = gw[s * 8 + m];
      }
      __syncwarp();
      unsigned first = 0, end = 0;  // bit j: row j starts / ends its skewer
#pragma unroll
      for (int j = 0; j < LG_PJ; ++j) {
        const int k = (row0 + 4 * j + rr) % n_per;
        first |= (unsigned)(k == 0) << j;
        end |= (unsigned)(k == n_per - 1) << j;
      }
      const float* hr = h + (size_t)(row0 + rr) * LG_N + 4 * c4;
      for (int c = 0; c < LG_NCH; ++c, ++g) {
        const uint32_t s = g % LG_STAGES;
        float4 v[LG_PJ];
        const int part = c / 4, ch = 32 * (c % 4);
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        if (part == 0) {
#pragma unroll
          for (int j = 0; j < LG_PJ; ++j)
            v[j] = *reinterpret_cast<const float4*>(hr + 4 * j * LG_N + ch);
        } else if (part == 1) {
#pragma unroll
          for (int j = 0; j < LG_PJ; ++j) {
            const float* p = hr + 4 * j * LG_N + ch;
            float4 az = zero;
            if (!((first >> j) & 1u)) az = f4_add(az, *reinterpret_cast<const float4*>(p - LG_N));
            if (!((end >> j) & 1u)) az = f4_add(az, *reinterpret_cast<const float4*>(p + LG_N));
            v[j] = az;
          }
        } else {
#pragma unroll
          for (int j = 0; j < LG_PJ; ++j) {
            const int r = LG_PR * warp + 4 * j + rr;
            float4 u[8];
#pragma unroll
            for (int m = 0; m < 8; ++m)
              u[m] = *reinterpret_cast<const float4*>(h + (size_t)sm.nb[r][m] * LG_N + ch +
                                                      4 * c4);
            float4 an = zero;
#pragma unroll
            for (int m = 0; m < 8; ++m) an = f4_fma(sm.g[r][m], u[m], an);
            v[j] = an;
          }
        }
        if (g >= LG_STAGES &&
            !lg_warp_wait(sm, &sm.empty[s], ((g / LG_STAGES) - 1) & 1u, err, 71, lane)) {
          ok = false;
          break;
        }
        if (tid == 0) {
          mbar_expect_tx(&sm.b_full[s], LG_OPF * sizeof(float));
          bulk_g2s(sm.b[s], wt + (size_t)c * LG_OPF, LG_OPF * sizeof(float), &sm.b_full[s]);
          last = (int)g;
        }
#pragma unroll
        for (int j = 0; j < LG_PJ; ++j)
          *reinterpret_cast<float4*>(&sm.a[s][lg_at_a(LG_PR * warp + 4 * j + rr, 4 * c4)]) = v[j];
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.full[s]);
      }
    }
  } else if (warp < LG_PW + 4) {
    // ---- epilogue -----------------------------------------------------------
    const int rs = warp & 3;
    uint32_t k = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, ++k) {
      const int tile = lg_tile(t, n_tiles, n_per);
      const uint32_t db = k & 1;
      if (!lg_warp_wait(sm, &sm.d_full[db], (k >> 1) & 1u, err, 72, lane)) break;
      tc_fence_after();
      const size_t m = (size_t)tile * 128 + 32 * rs;
      float(*tr)[LG_TW] = sm.t[rs];
#pragma unroll 1
      for (int j = 0; j < LG_N / 32; ++j) {
        float d[32];
        tmem_ld<32>(tmem + ((uint32_t)(32 * rs) << 16) + db * 128u + 32u * j, d);
        // through shared memory to 4 rows of 128 contiguous bytes per access
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<float4*>(&tr[lane][4 * q]) =
              make_float4(d[4 * q], d[4 * q + 1], d[4 * q + 2], d[4 * q + 3]);
        __syncwarp();
        const int c = 32 * j + 4 * (lane & 7);
        const float4 bb = *reinterpret_cast<const float4*>(bias + c);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int r = 4 * q + (lane >> 3);
          const float4 dd = *reinterpret_cast<const float4*>(&tr[r][4 * (lane & 7)]);
          const float4 res = *reinterpret_cast<const float4*>(h + (m + r) * LG_N + c);
          *reinterpret_cast<float4*>(out + (m + r) * LG_N + c) =
              make_float4(res.x + fmaxf(dd.x + bb.x, 0.f), res.y + fmaxf(dd.y + bb.y, 0.f),
                          res.z + fmaxf(dd.z + bb.z, 0.f), res.w + fmaxf(dd.w + bb.w, 0.f));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.d_empty[db]);
    }
  } else if (lane == 0) {
    // ---- MMA issue ------------------------------------------------------------
    uint32_t g = 0, k = 0;
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++k) {
      const uint32_t db = k & 1;
      if (k >= 2 && !lg_wait(sm, &sm.d_empty[db], ((k >> 1) - 1) & 1u, err, 73)) break;
      tc_fence_after();
      bool ok = true;
      for (int c = 0; c < LG_NCH; ++c, ++g) {
        const uint32_t s = g % LG_STAGES;
        if (!lg_wait(sm, &sm.full[s], (g / LG_STAGES) & 1u, err, 74) ||
            !lg_wait(sm, &sm.b_full[s], (g / LG_STAGES) & 1u, err, 75)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = smem_u32(sm.a[s]), sb = smem_u32(sm.b[s]);
#pragma unroll
        for (int kk = 0; kk < LG_KC / 8; ++kk) {
          const uint64_t ad = sdesc(sa + kk * 2 * LG_LBO_A, LG_LBO_A, LG_SBO);
          const uint64_t bd = sdesc(sb + kk * 2 * LG_LBO, LG_LBO, LG_SBO);
          mma_tf32(tmem + db * 128u, ad, bd, LG_IDESC, (c > 0 || kk > 0) ? 1u : 0u);
        }
        mma_commit(&sm.empty[s]);
        last = (int)g;
      }
      if (!ok) break;
      mma_commit(&sm.d_full[db]);
    }
  }
  // an early exit waits for what is in flight: the last MMA commit, the last
  // bulk copies
  if (lane == 0 && *(volatile int*)&sm.abort && last >= 0) {
    if (warp == LG_PW + 4) mbar_wait(&sm.empty[last % LG_STAGES], (last / LG_STAGES) & 1u);
    if (warp == 0)
      for (int k = max(0, last - LG_STAGES + 1); k <= last; ++k)
        mbar_wait(&sm.b_full[k % LG_STAGES], (k / LG_STAGES) & 1u);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, 256);
}

}  // namespace

bool layer_tc_usable(int M, int N, int K) { return N == LG_N && K == LG_K && M % 128 == 0; }

// out = h + relu([h | A_z h | A_n h] W + b) for a message-passing layer (TF32
// tensor cores); nbr, gw: the 8 neighbour skewers of every skewer and their
// weights; wt: scratch for W^T (LG_N x LG_K floats, 16-byte aligned), err:
// device error flag.
void launch_layer_tc(int M, int n_per, const float* h, const int* nbr, const float* gw,
                     const __nv_bfloat16* W, const float* bias, float* out, float* wt, int* err,
                     cudaStream_t st) {
  k_wt_f32<<<(LG_K * LG_N + 255) / 256, 256, 0, st>>>(W, wt);
  DS_CHECK_LAUNCH();
  DS_CUDA(cudaFuncSetAttribute(k_layer_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)LG_SMEM_BYTES));
  int dev = 0, sms = 0;
  DS_CUDA(cudaGetDevice(&dev));
  DS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int grid = std::max(1, std::min(M / 128, sms));
  k_layer_tc<<<grid, LG_THREADS, LG_SMEM_BYTES, st>>>(M, n_per, h, nbr, gw, wt, bias, out, err);
  DS_CHECK_LAUNCH();
}

}  // namespace ds
