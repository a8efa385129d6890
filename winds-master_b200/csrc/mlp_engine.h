// mlp_engine.h -- internal host side of the bound-circulation MLP (the C ABI
// is include/winds_mlp.h); shared with the wake engine, which runs the
// network's forward pass on its own stream for the Kutta-Joukowski guess.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "engine.h"
#include "winds_mlp.h"

namespace winds {

// Rows and the parts of a gradient.
struct MlpWork {
  DevBuf t, y, xraw, part;
  int ensure(long long n, bool train, cudaStream_t s);
  int ensure_parts(long long n, cudaStream_t s);
  void release();
};

// y [n] = network on the raw rows x [n][n_in] (one launch).
int mlp_forward(const winds_mlp *m, const float *x, long long n, float *y, cudaStream_t s);

// Device copies of the output scale and the base flag.
const float *mlp_out_scale_dev(const winds_mlp *m);
const float *mlp_base_dev(const winds_mlp *m);
int mlp_n_in(const winds_mlp *m);
int mlp_device(const winds_mlp *m);
unsigned *mlp_err_word(const winds_mlp *m);

}  // namespace winds
