// mlp_launch.h -- kernels of the bound-circulation MLP (one BF16 tcgen05 kernel
// for the whole network, forward or forward and backward; Adam).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace winds {

constexpr int kMlpWidth = 128;  // hidden width
constexpr int kMlpInPad = 16;   // input features padded to one K step of the MMA

// Offsets in the parameter vector (and in a CTA's gradient, with the sum of
// squared errors after it).
__host__ __device__ constexpr int mlp_off_w(int L) { return L == 0 ? 0 : 2176 + 16512 * (L - 1); }
__host__ __device__ constexpr int mlp_off_b(int L) { return 2048 + 16512 * L; }
constexpr long long kMlpOffW5 = 51712;
constexpr long long kMlpOffB5 = 51840;
constexpr long long kMlpNParam = 51841;
constexpr long long kMlpLoss = kMlpNParam;

// Parts of a gradient: weights per pair of tiles (W1, W2, W3, W4), the biases of
// the first three layers per tile of 128 rows, b4, w5, b5 and the sum of squared
// errors per 64 rows. The sums of a part and of the parts are in fixed orders.
constexpr long long kMlpPartW = 16 * 128 + 3 * 128 * 128;
constexpr long long kMlpPartHead = 2 * 128 + 2;
__host__ __device__ constexpr int mlp_part_w(int L) { return L == 0 ? 0 : 2048 + 16384 * (L - 1); }
int mlp_tiles(long long n);

// Rows x [.][n_in] (FP32, standardised as (x - shift) * scale), row r of n at
// idx[r] or r. Forward: y [n]. Gradient of 0.5 * mean((y - t)^2) with inv_n =
// 1 / n: its parts.
struct MlpNetArgs {
  const float *x, *shift, *scale;
  int n_in;
  const int *idx;
  long long n;
  const float *theta;
  const __nv_bfloat16 *wbf;
  float *y;
  const float *t;
  float inv_n;
  float *part_w, *part_b, *part_h;
  unsigned *err;
  unsigned long long wait_limit_ns;
};
cudaError_t launch_mlp_forward(const MlpNetArgs &g, int sms, cudaStream_t s);
cudaError_t launch_mlp_gradient(const MlpNetArgs &g, cudaStream_t s);

// loss = loss_scale * sum of squared errors, and either grad (not null) or one
// Adam step on theta and its BF16 copy.
struct MlpUpdateArgs {
  const float *part_w, *part_b, *part_h;
  int tiles;
  float *loss;
  float loss_scale;
  float *grad;
  float *theta;
  __nv_bfloat16 *theta_bf;
  float *m, *v;
  float lr, b1, b2, eps, wd, c1, c2;
};
cudaError_t launch_mlp_update(const MlpUpdateArgs &a, cudaStream_t s);
cudaError_t launch_mlp_to_bf16(const float *theta, __nv_bfloat16 *theta_bf, long long n,
                               cudaStream_t s);

}  // namespace winds
