// FP32 GEMMs and message passing of the learned network's training step (and
// of its inference where the tensor-core layers do not apply).
//
// Forward layer:   Z = [h | A_z h | A_n h] W + b,  h' = h + relu(Z)
// Backward layer:  dW = [h | A_z h | A_n h]^T dZ,  db = column sums of dZ,
//                  dh = dh' + [dZ | A_z dZ | A_n^T dZ] [W_0^T; W_1^T; W_2^T],
//                  dZ of the layer below = dh where its Z > 0
// (A_z is symmetric; the aggregation's adjoint acts on dZ before the GEMM, so
// the backward GEMM has the forward one's shape and writes [M x H] instead of
// [M x 3 H], and its epilogue takes in the residual and the relu's mask.)
//
// All arithmetic is FP32 (training's gradients are checked against an FP64
// oracle; TF32 would not do).  The GEMMs are bound by the FP32 pipe (128 FMAs
// per clock per SM): 128 x 128 tiles, 8 x 8 outputs per thread, packed FMAs
// (fma.f32x2 halves the issue slots of the same FMAs; the pairs (a, a) are made
// in registers: stored doubled in shared memory, their loads took 74% of the
// L1's wavefronts and held the FMA pipe at 56%).  Every output sums over k in
// ascending order, as a plain loop would.
// Measured at 262,144 rows and width 128 (25.8 GFLOP each): layers 487 us, weight
// gradients 459 us (64 x 64 tiles with 4 x 4 outputs: 985 and 1,050 us); the whole
// step 18.4 -> 8.0 ms.
#include <cub/cub.cuh>

#include <algorithm>

#include "ds_learned.h"

namespace ds {
namespace {

constexpr int BM = 128, BN = 128, BK = 16, GT = 256;
constexpr int LDA = BM + 4;  // floats per k of the A tile (16-byte rows, 2-way conflicts
                             // at most on the transposing stores)
constexpr size_t GEMM_SMEM = 2 * BK * (LDA + BN) * sizeof(float);

using f32x2 = unsigned long long;

__device__ __forceinline__ void fma2(f32x2& c, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

__device__ __forceinline__ float2 unpack(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

__device__ __forceinline__ f32x2 dup(float a) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}

// A thread's outputs: warp (wm, wn) of 4 x 2 has rows 32 wm .., columns 64 wn
// .., lane (lr, lc) of 4 x 8 in it rows row(i), columns col(u) .. + 3.
struct Frag {
  int r0, c0;
  __device__ Frag(int tid)
      : r0(32 * (tid >> 6) + 4 * ((tid & 31) >> 3)), c0(64 * ((tid >> 5) & 1) + 4 * (tid & 7)) {}
  __device__ int row(int i) const { return r0 + 16 * (i >> 2) + (i & 3); }
  __device__ int col(int u) const { return c0 + 32 * u; }
};

// One BK step of the CTA's tile: acc[i][j] += a_i (b_2j, b_2j+1).
__device__ __forceinline__ void tile_step(const float* As, const float* Bs, const Frag& f,
                                          f32x2 (&acc)[8][4]) {
#pragma unroll
  for (int k = 0; k < BK; ++k) {
    const float4 a0 = *reinterpret_cast<const float4*>(As + k * LDA + f.r0);
    const float4 a1 = *reinterpret_cast<const float4*>(As + k * LDA + f.r0 + 16);
    const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(Bs + k * BN + f.c0);
    const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(Bs + k * BN + f.c0 + 32);
    const f32x2 a[8] = {dup(a0.x), dup(a0.y), dup(a0.z), dup(a0.w),
                        dup(a1.x), dup(a1.y), dup(a1.z), dup(a1.w)};
    const f32x2 b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) fma2(acc[i][j], a[i], b[j]);
  }
}

struct LayerArgs {
  int M, H;
  const float *A0, *A1;  // the operand [A0 | A1]: M x H and M x 2 H
  const float* B;        // 3 H x H
  const float* bias;     // forward
  const float* res;      // forward: h;  backward: dh of the layer above
  const float* Zp;       // backward: Z of the layer below
  float* Z;              // forward: Z (or null);  backward: dZ of the layer below
  float* out;            // forward: h';  backward: dh (or null)
};

template <bool BWD>
__global__ void __launch_bounds__(GT, 2) k_layer(LayerArgs a) {
  extern __shared__ __align__(16) float gsm[];
  float* As = gsm;                  // [2][BK][LDA]
  float* Bs = gsm + 2 * BK * LDA;   // [2][BK][BN]
  const int tid = threadIdx.x;
  const Frag fr(tid);
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int H = a.H, K = 3 * H;
  f32x2 acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  float4 va[2], vb[2];
  auto load = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = tid + GT * q;
      const int m = m0 + (e >> 2), k = k0 + 4 * (e & 3);
      const float* p = k < H ? a.A0 + (size_t)m * H + k : a.A1 + (size_t)m * 2 * H + (k - H);
      va[q] = m < a.M ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
      const int n = n0 + 4 * (e & 31);
      vb[q] = n < H ? *reinterpret_cast<const float4*>(a.B + (size_t)(k0 + (e >> 5)) * H + n)
                    : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = tid + GT * q;
      float* d = As + buf * BK * LDA + 4 * (e & 3) * LDA + (e >> 2);
      d[0] = va[q].x;
      d[LDA] = va[q].y;
      d[2 * LDA] = va[q].z;
      d[3 * LDA] = va[q].w;
      *reinterpret_cast<float4*>(Bs + buf * BK * BN + (e >> 5) * BN + 4 * (e & 31)) = vb[q];
    }
  };
  load(0);
  store(0);
  __syncthreads();
  for (int k0 = 0, buf = 0; k0 < K; k0 += BK, buf ^= 1) {
    const bool more = k0 + BK < K;
    if (more) load(k0 + BK);
    tile_step(As + buf * BK * LDA, Bs + buf * BK * BN, fr, acc);
    if (more) store(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + fr.row(i);
    if (m >= a.M) continue;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int n = n0 + fr.col(u);
      if (n >= H) continue;
      const size_t o = (size_t)m * H + n;
      const float2 c0 = unpack(acc[i][2 * u]), c1 = unpack(acc[i][2 * u + 1]);
      const float4 r = *reinterpret_cast<const float4*>(a.res + o);
      if (BWD) {
        const float4 d = make_float4(r.x + c0.x, r.y + c0.y, r.z + c1.x, r.w + c1.y);
        const float4 z = *reinterpret_cast<const float4*>(a.Zp + o);
        if (a.out) *reinterpret_cast<float4*>(a.out + o) = d;
        *reinterpret_cast<float4*>(a.Z + o) =
            make_float4(z.x > 0.f ? d.x : 0.f, z.y > 0.f ? d.y : 0.f, z.z > 0.f ? d.z : 0.f,
                        z.w > 0.f ? d.w : 0.f);
      } else {
        const float4 b = *reinterpret_cast<const float4*>(a.bias + n);
        const float4 z = make_float4(c0.x + b.x, c0.y + b.y, c1.x + b.z, c1.y + b.w);
        if (a.Z) *reinterpret_cast<float4*>(a.Z + o) = z;
        *reinterpret_cast<float4*>(a.out + o) =
            make_float4(r.x + fmaxf(z.x, 0.f), r.y + fmaxf(z.y, 0.f), r.z + fmaxf(z.z, 0.f),
                        r.w + fmaxf(z.w, 0.f));
      }
    }
  }
}

// Partial products of dW [3 H x H] = [A0 | A1]^T D over rows [chunk z, chunk
// (z + 1)): CTA (column block, row block of dW, z); with the first row block also
// the partial column sums of D (after all chunks' products in `part`).
__global__ void __launch_bounds__(GT, 2) k_layer_grad(int M, int H, int chunk,
                                                      const float* __restrict__ A0,
                                                      const float* __restrict__ A1,
                                                      const float* __restrict__ D,
                                                      float* __restrict__ part) {
  extern __shared__ __align__(16) float gsm[];
  float* As = gsm;
  float* Bs = gsm + 2 * BK * LDA;
  const int tid = threadIdx.x;
  const Frag fr(tid);
  const int n0 = blockIdx.x * BN, k0 = blockIdx.y * BM, K = 3 * H;
  const int mb = blockIdx.z * chunk, me = min(M, mb + chunk);
  f32x2 acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  float4 va[2], vb[2], cs = make_float4(0.f, 0.f, 0.f, 0.f);  // cs: D's column sums
  auto load = [&](int mm) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = tid + GT * q, m = mm + (e >> 5);
      const int k = k0 + 4 * (e & 31), n = n0 + 4 * (e & 31);
      const float* p = k < H ? A0 + (size_t)m * H + k : A1 + (size_t)m * 2 * H + (k - H);
      va[q] = m < me && k < K ? *reinterpret_cast<const float4*>(p)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
      vb[q] = m < me && n < H ? *reinterpret_cast<const float4*>(D + (size_t)m * H + n)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = tid + GT * q;
      cs = make_float4(cs.x + vb[q].x, cs.y + vb[q].y, cs.z + vb[q].z, cs.w + vb[q].w);
      *reinterpret_cast<float4*>(As + buf * BK * LDA + (e >> 5) * LDA + 4 * (e & 31)) = va[q];
      *reinterpret_cast<float4*>(Bs + buf * BK * BN + (e >> 5) * BN + 4 * (e & 31)) = vb[q];
    }
  };
  load(mb);
  store(0);
  __syncthreads();
  for (int mm = mb, buf = 0; mm < me; mm += BK, buf ^= 1) {
    const bool more = mm + BK < me;
    if (more) load(mm + BK);
    tile_step(As + buf * BK * LDA, Bs + buf * BK * BN, fr, acc);
    if (more) store(buf ^ 1);
    __syncthreads();
  }
  float* P = part + (size_t)blockIdx.z * K * H;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = k0 + fr.row(i);
    if (k >= K) continue;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int n = n0 + fr.col(u);
      if (n >= H) continue;
      const float2 c0 = unpack(acc[i][2 * u]), c1 = unpack(acc[i][2 * u + 1]);
      *reinterpret_cast<float4*>(P + (size_t)k * H + n) = make_float4(c0.x, c0.y, c1.x, c1.y);
    }
  }
  if (blockIdx.y == 0) {  // the rows' eight classes in order
    *reinterpret_cast<float4*>(Bs + 4 * tid) = cs;
    __syncthreads();
    if (tid < BN && n0 + tid < H) {
      float t = 0.f;
      for (int w = 0; w < GT / 32; ++w) t += Bs[w * BN + tid];
      part[(size_t)gridDim.z * K * H + (size_t)blockIdx.z * H + n0 + tid] = t;
    }
  }
}

// Partial sums for small gradients, a thread per channel c of D [M x H]: out[k]
// = sum_m a[m][k] D[m][c] for the NK columns of a, then the sums of D's own
// columns (BIAS_D) or of a's (in thread c = k; !BIAS_D).  Thread groups of a CTA
// take rows in turn; one partial of (NK + 1) H floats per group.
template <int NK, bool BIAS_D>
__global__ void __launch_bounds__(512) k_small_grad(int M, int H, const float* __restrict__ a,
                                                    const float* __restrict__ D,
                                                    float* __restrict__ part) {
  const int G = blockDim.x / H, c = threadIdx.x % H, grp = threadIdx.x / H;
  const int stride = gridDim.x * G;
  float acc[NK], s = 0.f;
#pragma unroll
  for (int k = 0; k < NK; ++k) acc[k] = 0.f;
#pragma unroll 4
  for (int m = blockIdx.x * G + grp; m < M; m += stride) {
    const float d = D[(size_t)m * H + c];
#pragma unroll
    for (int k = 0; k < NK; ++k) acc[k] = fmaf(a[(size_t)m * NK + k], d, acc[k]);
    if (BIAS_D)
      s += d;
    else if (c < NK)
      s += a[(size_t)m * NK + c];
  }
  float* p = part + (size_t)(blockIdx.x * G + grp) * (NK + 1) * H;
#pragma unroll
  for (int k = 0; k < NK; ++k) p[(size_t)k * H + c] = acc[k];
  p[(size_t)NK * H + c] = s;
}

// Sums over the partials in order, one warp per value: lane l takes partials l,
// l + 32, ..., then a shuffle tree.  out[i] of len values; the partials lie
// `stride` apart; TRANS: value (k, c) = (i / H, i % H) goes to out[c NK + k].
__global__ void k_reduce_parts(int n_parts, int len, size_t stride, const float* __restrict__ part,
                               int H, int NK, float* __restrict__ out) {
  const int i = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= len) return;
  float s = 0.f;
  for (int p = lane; p < n_parts; p += 32) s += part[(size_t)p * stride + i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) out[NK ? (i % H) * NK + i / H : i] = s;
}

// The same with one thread per value and the partials in ascending order, for
// the large products (coalesced over the values).
__global__ void k_reduce_chunks(int n_parts, size_t len, const float* __restrict__ part,
                                float* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= len) return;
  float s = 0.f;
#pragma unroll 8
  for (int p = 0; p < n_parts; ++p) s += part[(size_t)p * len + i];
  out[i] = s;
}

// [A_z v | S v] per row, v [M x H]: A_z v_i = v_{i-1} + v_{i+1} along the skewer,
// S v = sum over the skewer's list of weight x the row of the listed skewer at
// the same z index.  Lists: 8 entries per skewer (ptr null: the neighbours, S =
// A_n) or CSR (ptr: the skewers that name this one, S = A_n^T).  Four channels
// per thread.
__global__ void k_aggregate(int n, int n_per, int H, const float* __restrict__ v,
                            const int* __restrict__ ptr, const int* __restrict__ idx,
                            const float* __restrict__ w, float* __restrict__ out) {
  const int H4 = H >> 2;
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (size_t)n * H4) return;
  const int i = (int)(q / H4), c4 = (int)(q % H4);
  const int s = i / n_per, k = i % n_per;
  const float4* v4 = reinterpret_cast<const float4*>(v);
  float4 az = make_float4(0.f, 0.f, 0.f, 0.f);
  auto add = [&](const float4 u) {
    az = make_float4(az.x + u.x, az.y + u.y, az.z + u.z, az.w + u.w);
  };
  if (k > 0) add(v4[q - H4]);
  if (k + 1 < n_per) add(v4[q + H4]);
  float4 an = make_float4(0.f, 0.f, 0.f, 0.f);
  auto mac = [&](int e) {
    const float g = w[e];
    const float4 u = v4[((size_t)idx[e] * n_per + k) * H4 + c4];
    an = make_float4(fmaf(g, u.x, an.x), fmaf(g, u.y, an.y), fmaf(g, u.z, an.z),
                     fmaf(g, u.w, an.w));
  };
  if (!ptr) {
#pragma unroll
    for (int m = 0; m < 8; ++m) mac(s * 8 + m);
  } else {
    const int e1 = ptr[s + 1];
#pragma unroll 4
    for (int e = ptr[s]; e < e1; ++e) mac(e);
  }
  float4* o = reinterpret_cast<float4*>(out + (size_t)i * 2 * H);
  o[c4] = az;
  o[H4 + c4] = an;
}

// dh4 = dY W_o^T (4 outputs) and dZ4 = dh4 where Z4 > 0.
__global__ void k_head_bwd(int n, int H, const float* __restrict__ dY,
                           const __nv_bfloat16* __restrict__ W, const float* __restrict__ Z,
                           float* __restrict__ dh, float* __restrict__ dZ) {
  const int H4 = H >> 2;
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (size_t)n * H4) return;
  const int i = (int)(q / H4), c = 4 * (int)(q % H4);
  const float4 y = reinterpret_cast<const float4*>(dY)[i];
  float d[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    float s = y.x * __bfloat162float(W[(c + u) * 4]);
    s = fmaf(y.y, __bfloat162float(W[(c + u) * 4 + 1]), s);
    s = fmaf(y.z, __bfloat162float(W[(c + u) * 4 + 2]), s);
    d[u] = fmaf(y.w, __bfloat162float(W[(c + u) * 4 + 3]), s);
  }
  const float4 z = reinterpret_cast<const float4*>(Z)[q];
  reinterpret_cast<float4*>(dh)[q] = make_float4(d[0], d[1], d[2], d[3]);
  reinterpret_cast<float4*>(dZ)[q] =
      make_float4(z.x > 0.f ? d[0] : 0.f, z.y > 0.f ? d[1] : 0.f, z.z > 0.f ? d[2] : 0.f,
                  z.w > 0.f ? d[3] : 0.f);
}

// The layer weights [3 H x H] as FP32, for the forward GEMM as they are, for
// the backward one each H x H block transposed.
__global__ void k_layer_weights(int H, bool trans, const __nv_bfloat16* __restrict__ W,
                                float* __restrict__ B) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * H * H) return;
  const int k = i / H, n = i % H, p = k / H, j = k % H;
  B[i] = __bfloat162float(trans ? W[(size_t)(p * H + n) * H + j] : W[i]);
}

// Reverse neighbour lists: the skewers that name skewer t, in ascending order.
__global__ void k_rev_count(int n, const int* __restrict__ nbr, const float* __restrict__ g,
                            int* __restrict__ cnt) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n && g[e] != 0.f) atomicAdd(&cnt[nbr[e]], 1);
}

__global__ void k_rev_fill(int n, const int* __restrict__ nbr, const float* __restrict__ g,
                           const int* __restrict__ ptr, int* __restrict__ cnt,
                           int* __restrict__ src) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n && g[e] != 0.f) src[ptr[nbr[e]] + atomicSub(&cnt[nbr[e]], 1) - 1] = e;
}

// Writes the skewer and weight of every entry in ascending order of the entry numbers
// (it does not depend on the atomics): a warp per list, each entry at its rank.  The
// lists have some 8 entries; where many skewers share a line of sight, 8 of them are
// named by all (a training step of 4,000 such skewers x 4 pixels: 166 ms with one
// thread's insertion sort per list, 7.5 here).
__global__ void k_rev_sort(int n_sk, const int* __restrict__ ptr, const int* __restrict__ src,
                           const float* __restrict__ g, int* __restrict__ idx,
                           float* __restrict__ w) {
  const int s = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  if (s >= n_sk) return;
  const int a = ptr[s], b = ptr[s + 1];
  for (int i = a + (threadIdx.x & 31); i < b; i += 32) {
    const int v = src[i];
    int rank = 0;
    for (int j = a; j < b; ++j) rank += src[j] < v;
    idx[a + rank] = v / 8;
    w[a + rank] = g[v];
  }
}

inline unsigned grid1(size_t n, int nt = 256) { return (unsigned)((n + nt - 1) / nt); }

template <bool BWD>
void launch(const LayerArgs& a, cudaStream_t st) {
  DS_CUDA(cudaFuncSetAttribute(k_layer<BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)GEMM_SMEM));
  k_layer<BWD><<<dim3((a.M + BM - 1) / BM, (a.H + BN - 1) / BN), GT, GEMM_SMEM, st>>>(a);
  DS_CHECK_LAUNCH();
}

}  // namespace

// Rows per chunk of a layer's weight gradient: two CTAs per SM over all chunks
// and output tiles in one wave (equal chunks; a last wave of a few CTAs cost a
// third of the kernel), whole steps of BK rows.
int layer_grad_chunk(int M, int H, int sms) {
  const int tiles = ((3 * H + BM - 1) / BM) * ((H + BN - 1) / BN);
  const int chunks = std::max(1, 2 * sms / tiles);
  return std::max(BK, ((M + chunks - 1) / chunks + BK - 1) / BK * BK);
}

size_t layer_grad_parts(int M, int H, int sms) {
  const int chunk = layer_grad_chunk(M, H, sms);
  return (size_t)((M + chunk - 1) / chunk) * (3 * (size_t)H + 1) * H;
}

// h' = h + relu(Z), Z = [h | A_z h | A_n h] W + b: agg receives the aggregated
// columns [M x 2 H] (kept for the backward pass), wf is scratch for W (3 H x H).
void layer_forward(int M, int n_per, int H, const float* h, const int* nbr, const float* g,
                   const __nv_bfloat16* W, const float* bias, float* agg, float* wf, float* Z,
                   float* out, cudaStream_t st) {
  k_layer_weights<<<grid1(3 * (size_t)H * H), 256, 0, st>>>(H, false, W, wf);
  DS_CHECK_LAUNCH();
  k_aggregate<<<grid1((size_t)M * (H / 4)), 256, 0, st>>>(M, n_per, H, h, nullptr, nbr, g, agg);
  DS_CHECK_LAUNCH();
  LayerArgs a{M, H, h, agg, wf, bias, h, nullptr, Z, out};
  launch<false>(a, st);
}

// The layer's gradients and dh, dZ of the layer below (see the head of the
// file).  dZ: in, this layer's; dZ_below: out; dh: in, of the layer above, out
// (unless last), of the layer below.  agg: as kept by layer_forward; aggT:
// scratch M x 2 H.
void layer_backward(int M, int n_per, int H, int sms, const float* h, const float* agg,
                    const RevLists& rev, const __nv_bfloat16* W, const float* Z_below,
                    const float* dZ, float* dZ_below, float* dh, bool last, float* aggT, float* wf,
                    float* part, float* dW, float* db, cudaStream_t st) {
  const int chunk = layer_grad_chunk(M, H, sms), chunks = (M + chunk - 1) / chunk;
  DS_CUDA(cudaFuncSetAttribute(k_layer_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)GEMM_SMEM));
  k_layer_grad<<<dim3((H + BN - 1) / BN, (3 * H + BM - 1) / BM, chunks), GT, GEMM_SMEM, st>>>(
      M, H, chunk, h, agg, dZ, part);
  DS_CHECK_LAUNCH();
  const size_t len = 3 * (size_t)H * H;
  k_reduce_chunks<<<grid1(len), 256, 0, st>>>(chunks, len, part, dW);
  DS_CHECK_LAUNCH();
  k_reduce_parts<<<grid1(32 * (size_t)H), 256, 0, st>>>(chunks, H, H, part + chunks * len, H, 0,
                                                        db);
  DS_CHECK_LAUNCH();
  k_layer_weights<<<grid1(len), 256, 0, st>>>(H, true, W, wf);
  DS_CHECK_LAUNCH();
  k_aggregate<<<grid1((size_t)M * (H / 4)), 256, 0, st>>>(M, n_per, H, dZ, rev.ptr.p, rev.idx.p,
                                                          rev.w.p, aggT);
  DS_CHECK_LAUNCH();
  LayerArgs a{M, H, dZ, aggT, wf, nullptr, dh, Z_below, dZ_below, last ? nullptr : dh};
  launch<true>(a, st);
}

void head_backward(int n, int H, const float* dY, const __nv_bfloat16* W, const float* Z,
                   float* dh, float* dZ, cudaStream_t st) {
  k_head_bwd<<<grid1((size_t)n * (H / 4)), 256, 0, st>>>(n, H, dY, W, Z, dh, dZ);
  DS_CHECK_LAUNCH();
}

// CTAs of the small gradients: 4 of 512 threads per SM (bound by reading D).
static int small_groups(int H, int sms) { return 4 * sms * (512 / H); }

size_t small_grad_parts(int H, int sms) { return (size_t)small_groups(H, sms) * 12 * H; }

// dW_o [H x 4] = h^T dY and db_o.
void head_grad(int M, int H, int sms, const float* h, const float* dY, float* part, float* dW,
               float* db, cudaStream_t st) {
  const int G = 512 / H, parts = small_groups(H, sms);
  k_small_grad<4, false><<<parts / G, G * H, 0, st>>>(M, H, dY, h, part);
  DS_CHECK_LAUNCH();
  k_reduce_parts<<<grid1(32 * 4 * (size_t)H), 256, 0, st>>>(parts, 4 * H, (size_t)5 * H, part, H,
                                                            4, dW);
  DS_CHECK_LAUNCH();
  k_reduce_parts<<<1, 128, 0, st>>>(parts, 4, (size_t)5 * H, part + 4 * (size_t)H, H, 0, db);
  DS_CHECK_LAUNCH();
}

// dW_in [11 x H] = X^T dZ and db_in.
void embed_grad(int M, int H, int sms, const float* X, const float* dZ, float* part, float* dW,
                float* db, cudaStream_t st) {
  const int G = 512 / H, parts = small_groups(H, sms);
  k_small_grad<F_IN, true><<<parts / G, G * H, 0, st>>>(M, H, X, dZ, part);
  DS_CHECK_LAUNCH();
  const size_t stride = (size_t)(F_IN + 1) * H;
  k_reduce_parts<<<grid1(32 * F_IN * (size_t)H), 256, 0, st>>>(parts, F_IN * H, stride, part, H, 0,
                                                               dW);
  DS_CHECK_LAUNCH();
  k_reduce_parts<<<grid1(32 * (size_t)H), 256, 0, st>>>(parts, H, stride, part + F_IN * (size_t)H,
                                                        H, 0, db);
  DS_CHECK_LAUNCH();
}

// The reverse lists of nbr (8 per skewer; entries of weight 0 are left out).
void build_rev_lists(int n_sk, const int* nbr, const float* g, RevLists& rev, cudaStream_t st) {
  const int n = n_sk * 8;
  rev.ptr.alloc(n_sk + 1);
  rev.cnt.alloc(n_sk + 1);
  rev.src.alloc(n);
  rev.idx.alloc(n);
  rev.w.alloc(n);
  DS_CUDA(cudaMemsetAsync(rev.cnt.p, 0, rev.cnt.bytes(), st));
  k_rev_count<<<grid1(n), 256, 0, st>>>(n, nbr, g, rev.cnt.p);
  DS_CHECK_LAUNCH();
  size_t bytes = 0;
  DS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, rev.cnt.p, rev.ptr.p, n_sk + 1, st));
  if (rev.tmp.n < bytes) rev.tmp.alloc(bytes);
  DS_CUDA(cub::DeviceScan::ExclusiveSum(rev.tmp.p, bytes, rev.cnt.p, rev.ptr.p, n_sk + 1, st));
  k_rev_fill<<<grid1(n), 256, 0, st>>>(n, nbr, g, rev.ptr.p, rev.cnt.p, rev.src.p);
  DS_CHECK_LAUNCH();
  k_rev_sort<<<grid1(32 * (size_t)n_sk), 256, 0, st>>>(n_sk, rev.ptr.p, rev.src.p, g, rev.idx.p,
                                                       rev.w.p);
  DS_CHECK_LAUNCH();
}

}  // namespace ds
