// The learned warm start and per-skewer preconditioner (learned.cu), and the
// skewer-band preconditioner of the mixed-precision solver (skewer_pc.cu).
#pragma once

#include <cuda_bf16.h>

#include <atomic>

#include "ds_internal.cuh"

namespace ds {

constexpr int F_IN = 11;      // input features per pixel
constexpr int N_LAYERS = 4;   // message-passing layers

// The skewers that name each skewer as a neighbour (learned_gemm.cu), CSR.
struct RevLists {
  DevBuf<int> ptr, cnt, src, idx;
  DevBuf<float> w;
  DevBuf<unsigned char> tmp;
};

struct LearnedNet {
  struct Slot {
    size_t off = 0, rows = 0, cols = 0;
    bool bias = false;
  };
  ds_context* ctx;
  int H, B, NO = 0;
  KernelConsts kc;
  size_t n_params = 0;
  Slot W_in, b_in, W_l[N_LAYERS], b_l[N_LAYERS], W_o, b_o;
  DevBuf<float> params, grads, adam_m, adam_v;
  DevBuf<unsigned short> wbf;  // BF16 copy of the parameters (forward weights)
  long long step = 0;
  // per-geometry work space
  const double* rec_cur = nullptr;  // records of the last forward (device)
  size_t n_cur = 0;
  int nsk_cur = 0;
  DevBuf<int> nbr;
  DevBuf<double2> skxy;  // (x, y) per skewer
  DevBuf<float> gw, X, h[N_LAYERS + 1], Y, wf;
  DevBuf<float> agg[N_LAYERS];  // [A_z h | A_n h] per layer (without training: the first alone)
  // training
  DevBuf<float> Z[N_LAYERS + 1], dY, dh, dZ, dZ2, aggT, part;
  RevLists rev;
  DevBuf<double> dpart;
  // inference: message-passing layers on the tensor cores (learned_tc.cu)
  bool tc_infer = true;
  bool tc_active = false;
  DevBuf<float> wt;   // W^T of the layer in flight (FP32)
  DevBuf<int> tc_err;

  LearnedNet(ds_context* c, int hidden, int band, const KernelConsts& k, unsigned seed);
  void sync_weights();
  void ensure(int n_sk, int n_per);
  void ensure_train();
  // records: W-form records (x, y, z, w, w d) of n_sk skewers x n_per pixels,
  // skewer-contiguous, on the device
  // train: keeps Z and the aggregated activations for backward()
  void forward(int n_sk, int n_per, const double* rec, bool train);
  void outputs(int n_sk, int n_per, double* y0, float* Lrows);
  void loss_and_grad(int n_sk, int n_per, const double* rec, const double* ystar,
                     const float* probe, float wx, float wp, double* losses);
  void backward(int n_sk, int n_per);
  void adam_step(float lr);
};

// Band preconditioner M^-1 = L L^T of an operator over blocks of `n_per`
// slots (FP32 L rows of bandwidth `band`, indexed by slot): per skewer (slot
// = record, blocks of n_per consecutive records) or per cluster of
// neighbouring skewers (crec: the record of each slot, -1 on padding).
bool layer_tc_usable(int M, int N, int K);
void launch_layer_tc(int M, int n_per, const float* h, const int* nbr, const float* gw,
                     const __nv_bfloat16* W, const float* bias, float* out, float* wt, int* err,
                     cudaStream_t st);

// FP32 layers, forward and backward (learned_gemm.cu).
size_t layer_grad_parts(int M, int H, int sms);
size_t small_grad_parts(int H, int sms);
void layer_forward(int M, int n_per, int H, const float* h, const int* nbr, const float* g,
                   const __nv_bfloat16* W, const float* bias, float* agg, float* wf, float* Z,
                   float* out, cudaStream_t st);
void layer_backward(int M, int n_per, int H, int sms, const float* h, const float* agg,
                    const RevLists& rev, const __nv_bfloat16* W, const float* Z_below,
                    const float* dZ, float* dZ_below, float* dh, bool last, float* aggT, float* wf,
                    float* part, float* dW, float* db, cudaStream_t st);
void head_backward(int n, int H, const float* dY, const __nv_bfloat16* W, const float* Z,
                   float* dh, float* dZ, cudaStream_t st);
void head_grad(int M, int H, int sms, const float* h, const float* dY, float* part, float* dW,
               float* db, cudaStream_t st);
void embed_grad(int M, int H, int sms, const float* X, const float* dZ, float* part, float* dW,
                float* db, cudaStream_t st);
void build_rev_lists(int n_sk, const int* nbr, const float* g, RevLists& rev, cudaStream_t st);

inline unsigned long long next_pc_serial() {
  static std::atomic<unsigned long long> n{0};
  return ++n;
}

struct SkewerPC {
  // identity for what is built from it (an address can come back)
  const unsigned long long serial = next_pc_serial();
  int n_sk = 0, n_per = 0, band = 0;  // blocks, slots per block, bandwidth
  DevBuf<float> L;    // band + 1 planes of n_sk n_per slots: L[k][k - m] at plane m
  DevBuf<int> crec;   // record of each slot (empty: slot = record)
  int n_fallback = 0;  // cluster factor: columns that fell back to Jacobi
  // skewers per block and the skewers of each block (g per block, -1 on
  // padding; empty: block b is skewer b, g = 1)
  int g = 1;
  DevBuf<int> bsk;
};

}  // namespace ds

struct ds_learned {
  std::unique_ptr<ds::LearnedNet> net;
};
