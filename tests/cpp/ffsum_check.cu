// The persistent and batched solves' sums and scalars (csrc/ds_ffsum.cuh) on the
// device, against the same in exact or FP64 arithmetic on the host.  Prints "name error bound" lines.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "ds_ffsum.cuh"

using namespace ds;

constexpr int NT = 512;

__global__ void k_sums(const float2* v, const float2* w, double* out) {
  __shared__ float2 sm[2 * (NT / 32)];
  const int t = threadIdx.x, base = blockIdx.x * NT;
  const ff a{v[base + t].x, v[base + t].y}, b{w[base + t].x, w[base + t].y};
  const double s = block_sum2<NT, true>(a, b, sm);
  if (t == 0 || t == 16) out[3 * blockIdx.x + (t >> 4)] = s;
  __syncthreads();
  const double one = block_sum2<NT, false>(a, ff{0.f, 0.f}, sm);
  if (t == 0) out[3 * blockIdx.x + 2] = one;
}

__global__ void k_quotients(int n, const double* a, const double* b, float2* q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const ff r = quotient_ff(a[i], b[i]);
  q[i] = make_float2(r.h, r.l);
}

// The update test at |r|^2 = rr[i] after an update at |r| = 1 (scaled by `unit`).
__global__ void k_norms(int n, const double* rr, double unit, double delta, double tol, int* due,
                        double* back) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  MixedState s{};
  s.max_iter = 100;
  s.delta = delta;
  s.tol_norm_b = tol * unit;
  s.rmax = s.rbest = unit;
  s.rz = 0.75 * unit * unit;
  FastState f;
  fast_from(f, s, unit);
  const double sr = f.sr;
  fast_norm(f, s, 1, rr[i] * (unit * sr) * (unit * sr));
  due[i] = s.need_update;
  f.pq = f.rz;
  f.alpha = ff{1.f, 0.f};
  fast_to(f, s);
  back[i] = s.rnorm;
}

// A tile's dot product as the batched step forms it: 8 groups of 16 rows.
__global__ void k_tile(const float* x, const float* y, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  f3 total{0.f, 0.f, 0.f};
  for (int g = 0; g < 8; ++g) {
    f3 v{0.f, 0.f, 0.f};
    for (int k = 0; k < 16; ++k) {
      const size_t e = (size_t)i * 128 + 16 * g + k;
      f3_acc_prod(v, x[e], y[e]);
    }
    f3_add(total, v);
  }
  out[i] = f3_double(total);
}

template <class T>
T* up(const std::vector<T>& v) {
  T* p = nullptr;
  cudaMalloc(&p, v.size() * sizeof(T));
  cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  return p;
}

template <class T>
std::vector<T> down(const T* p, size_t n) {
  std::vector<T> v(n);
  if (cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost) != cudaSuccess) {
    printf("CUDA error\n");
    exit(1);
  }
  return v;
}

int main() {
  std::mt19937_64 rng(1);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  const double u53 = ldexp(1.0, -53);
  // Block sums.  Half the blocks have values in one lane of each warp alone, whose
  // float-pair tree adds zeros: their sums are FP64's, 4 additions of 2^-53 each and
  // one of the two halves.  The others': 5 float-pair additions of 2^-45 at most.
  const int B = 64;
  std::vector<float2> v(B * NT), w(B * NT);
  for (int b = 0; b < B; ++b)
    for (int t = 0; t < NT; ++t) {
      const bool in = b < B / 2 ? t % 32 == 0 : true;
      auto draw = [&] {
        const double x = in ? (U(rng) - (b % 2 ? 0.5 : 0.0)) * exp(4 * U(rng)) : 0.0;
        const float h = (float)x;
        return make_float2(h, (float)(x - (double)h));
      };
      v[b * NT + t] = draw();
      w[b * NT + t] = draw();
    }
  double *dsum = up(std::vector<double>(3 * B));
  k_sums<<<B, NT>>>(up(v), up(w), dsum);
  const auto s = down(dsum, 3 * B);
  double e64 = 0, eff = 0;
  for (int b = 0; b < B; ++b)
    for (int k = 0; k < 3; ++k) {
      const std::vector<float2>& x = k == 1 ? w : v;
      long double sum = 0, mag = 0;
      for (int t = 0; t < NT; ++t) {
        const long double a = (long double)x[b * NT + t].x + x[b * NT + t].y;
        sum += a;
        mag += fabsl(a);
      }
      double& e = b < B / 2 ? e64 : eff;
      e = fmax(e, (double)(fabsl(s[3 * b + k] - sum) / mag));
    }
  printf("warps_up %g %g\n", e64, 5 * u53);
  printf("threads_up %g %g\n", eff, 5 * ldexp(1.0, -45) + 5 * u53);
  // Quotients: the first digit to 2^-23, the second 2^-23 of that (with the rounding
  // of the remainder's conversion and of the divisor's, 2^-24 each).
  const int n = 4096;
  std::vector<double> a(n), b(n);
  for (int i = 0; i < n; ++i) {
    a[i] = (U(rng) - 0.3) * exp(30 * (U(rng) - 0.5));
    b[i] = (0.1 + U(rng)) * exp(30 * (U(rng) - 0.5));
  }
  float2* dq = up(std::vector<float2>(n));
  k_quotients<<<n / 256, 256>>>(n, up(a), up(b), dq);
  const auto q = down(dq, n);
  double eq = 0;
  for (int i = 0; i < n; ++i) {
    const long double ref = (long double)a[i] / b[i];
    eq = fmax(eq, (double)fabsl(((long double)q[i].x + q[i].y - ref) / ref));
  }
  printf("quotient %g %g\n", eq, ldexp(1.0, -45));
  // A tile's sum in three floats: 128^3 2^-72 of the terms' magnitudes and the three
  // roundings to FP64.
  const int nt = 1024;
  std::vector<float> x((size_t)nt * 128), y(x.size());
  for (size_t i = 0; i < x.size(); ++i) {
    x[i] = (float)((U(rng) - 0.5) * exp(6 * U(rng)));
    y[i] = i % 3 ? (float)((U(rng) - 0.3) * exp(6 * U(rng))) : x[i];
  }
  double* dt = up(std::vector<double>(nt));
  k_tile<<<nt / 128, 128>>>(up(x), up(y), dt);
  const auto tiles = down(dt, nt);
  double et = 0;
  for (int i = 0; i < nt; ++i) {
    // the exact products' sum by long double (64 bits or more), compensated
    long double sum = 0, low = 0, mag = 0;
    for (int k = 0; k < 128; ++k) {
      const long double p = (long double)x[(size_t)i * 128 + k] * y[(size_t)i * 128 + k];
      const long double t = sum + p, bb = t - sum;
      low += (sum - (t - bb)) + (p - bb);
      sum = t;
      mag += fabsl(p);
    }
    et = fmax(et, (double)(fabsl((tiles[i] - sum) - low) / mag));
  }
  printf("tile %g %g\n", et, ldexp(1.0, 21 - 72) + 3 * u53);
  // The update test 2^-46 on either side of delta^2 and of tol^2, in three units.
  for (double unit : {1.0, 1e-17, 1e12}) {
    const double delta = 1e-4, tol = 3e-3, d = ldexp(1.0, -46);
    const std::vector<double> rr{delta * delta * (1 + d), delta * delta * (1 - d)};
    const std::vector<double> rt{tol * tol * (1 + d), tol * tol * (1 - d)};
    int wrong = 0;
    double er = 0;
    for (int k = 0; k < 2; ++k) {
      const auto& r = k ? rt : rr;
      int* due = up(std::vector<int>(2));
      double* back = up(std::vector<double>(2));
      k_norms<<<1, 2>>>(2, up(r), unit, delta, k ? tol : 0.0, due, back);
      const auto h = down(due, 2);
      const auto bk = down(back, 2);
      wrong += h[0] != 0;
      wrong += h[1] != 1;
      for (int i = 0; i < 2; ++i) er = fmax(er, fabs(bk[i] / (sqrt(r[i]) * unit) - 1));
    }
    printf("update_test %d 0\n", wrong);
    printf("norm %g %g\n", er, 8 * u53);
  }
  return 0;
}
