// mlp_engine.cu -- host side of the bound-circulation MLP: parameters,
// forward / backward launch sequences, Adam training, C ABI (winds_mlp.h).
//
// One training step on a batch of n rows is two launches: mlp_net (forward and
// backward of every 128 rows, gradients summed per CTA) and mlp_update (the
// CTAs' gradients summed in order, which keeps the result deterministic, and
// Adam on the FP32 master vector with its BF16 copy). Inference is one.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "bs_launch.h"
#include "host_stage.h"
#include "mlp_engine.h"
#include "mlp_launch.h"

struct winds_mlp {
  int dev = 0;
  int n_in = 0;
  int sms = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  winds::DevBuf theta, theta_bf, grad, mom, vel, shift, scale, err, loss, lossbuf, idx;
  winds::DevBuf Xall, Tall;
  float out_scale = 1.f;
  int base = 0;  // start value the output is added to (winds_mlp_set_base)
  float h_shift[16], h_scale[16];
  long long adam_t = 0;
  winds::MlpWork w;
  double train_ms = 0.0;
  long long train_steps = 0;
};

namespace winds {
namespace {

constexpr int W = kMlpWidth;
constexpr long long kNParam = kMlpNParam;
constexpr int kInK[4] = {kMlpInPad, W, W, W};  // input width of each layer

template <class T>
T *P(DevBuf &b) {
  return static_cast<T *>(b.p);
}
template <class T>
const T *P(const DevBuf &b) {
  return static_cast<const T *>(b.p);
}

long long cdiv(long long a, long long b) { return (a + b - 1) / b; }

// Host to device on the model's stream: a plain cudaMemcpy from pageable memory
// may return before the data is on the device, and kernels on a non-blocking
// stream do not wait for it. src outlives the copy's staging, as the callers
// synchronise before they let go of it.
cudaError_t upload(void *dst, const void *src, size_t bytes, cudaStream_t s) {
  return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
}

MlpNetArgs net_args(const winds_mlp *m, const float *x, long long n) {
  MlpNetArgs g;
  std::memset(&g, 0, sizeof(g));
  g.x = x;
  g.shift = static_cast<const float *>(m->shift.p);
  g.scale = static_cast<const float *>(m->scale.p);
  g.n_in = m->n_in;
  g.n = n;
  g.theta = static_cast<const float *>(m->theta.p);
  g.wbf = static_cast<const __nv_bfloat16 *>(m->theta_bf.p);
  g.err = static_cast<unsigned *>(m->err.p);
  g.wait_limit_ns = default_wait_limit_ns();
  return g;
}

int check_err(winds_mlp *m) {
  unsigned word = 0;
  cudaError_t e = cudaMemcpy(&word, m->err.p, sizeof(word), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_fail(e, "mlp error word");
  if (word) {
    cudaMemset(m->err.p, 0, sizeof(unsigned));
    return fail(word & kErrWaitTimeout ? WINDS_BS_ERR_TIMEOUT : WINDS_BS_ERR_CUDA,
                "mlp kernels reported error word 0x%x", word);
  }
  return WINDS_BS_OK;
}

// Gradient of the rows x (those of idx, when given) with targets t, in parts for
// launch_mlp_update(u) to sum, which puts 0.5 * mean squared error in loss.
int gradient(winds_mlp *m, const float *x, const float *t, const int *idx, long long n, float *loss,
             MlpUpdateArgs *u, cudaStream_t s) {
  MlpNetArgs g = net_args(m, x, n);
  g.t = t;
  g.idx = idx;
  g.inv_n = (float)(1.0 / (double)n);
  const int tiles = mlp_tiles(n);
  g.part_w = P<float>(m->w.part);
  g.part_b = g.part_w + (tiles + 1) / 2 * kMlpPartW;
  g.part_h = g.part_b + tiles * 3LL * W;
  std::memset(u, 0, sizeof(*u));
  u->part_w = g.part_w, u->part_b = g.part_b, u->part_h = g.part_h;
  u->tiles = tiles;
  u->loss = loss;
  u->loss_scale = (float)(0.5 / (double)n);
  const cudaError_t e = launch_mlp_gradient(g, s);
  return e == cudaSuccess ? WINDS_BS_OK : cuda_fail(e, "mlp gradient");
}

int upload_inputs(winds_mlp *m, const float *x, long long n, cudaStream_t s) {
  const cudaError_t e = upload(m->w.xraw.p, x, (size_t)n * m->n_in * sizeof(float), s);
  return e == cudaSuccess ? WINDS_BS_OK : cuda_fail(e, "mlp input upload");
}

int adam_step(winds_mlp *m, const winds_mlp_train_params &p, MlpUpdateArgs u, cudaStream_t s) {
  ++m->adam_t;
  u.theta = P<float>(m->theta);
  u.theta_bf = P<__nv_bfloat16>(m->theta_bf);
  u.m = P<float>(m->mom);
  u.v = P<float>(m->vel);
  u.lr = p.lr, u.b1 = p.beta1, u.b2 = p.beta2, u.eps = p.eps, u.wd = p.weight_decay;
  u.c1 = (float)(1.0 - std::pow((double)p.beta1, (double)m->adam_t));
  u.c2 = (float)(1.0 - std::pow((double)p.beta2, (double)m->adam_t));
  const cudaError_t e = launch_mlp_update(u, s);
  return e == cudaSuccess ? WINDS_BS_OK : cuda_fail(e, "mlp adam");
}

}  // namespace

int MlpWork::ensure_parts(long long n, cudaStream_t s) {
  const long long tiles = mlp_tiles(n);
  return part.ensure(((tiles + 1) / 2 * kMlpPartW + tiles * (3 * W + 2 * kMlpPartHead)) * sizeof(float), s);
}

int MlpWork::ensure(long long n, bool train, cudaStream_t s) {
  int rc;
  if ((rc = t.ensure(n * 4, s)) || (rc = y.ensure(n * 4, s)) || (rc = xraw.ensure(n * 16 * 4, s)))
    return rc;
  return train ? ensure_parts(n, s) : WINDS_BS_OK;
}

void MlpWork::release() {
  for (DevBuf *b : {&t, &y, &xraw, &part}) b->release();
}

int mlp_forward(const winds_mlp *m, const float *x, long long n, float *y, cudaStream_t s) {
  MlpNetArgs g = net_args(m, x, n);
  g.y = y;
  const cudaError_t e = launch_mlp_forward(g, m->sms, s);
  return e == cudaSuccess ? WINDS_BS_OK : cuda_fail(e, "mlp forward");
}

// out_scale and the base flag on the device (after the 16 input scales), read
// when a captured step replays
const float *mlp_out_scale_dev(const winds_mlp *m) { return static_cast<const float *>(m->scale.p) + 16; }
const float *mlp_base_dev(const winds_mlp *m) { return static_cast<const float *>(m->scale.p) + 17; }
int mlp_n_in(const winds_mlp *m) { return m->n_in; }
int mlp_device(const winds_mlp *m) { return m->dev; }
unsigned *mlp_err_word(const winds_mlp *m) { return static_cast<unsigned *>(m->err.p); }

}  // namespace winds

using namespace winds;

extern "C" {

int winds_mlp_create(const winds_mlp_config *cfg, winds_mlp **out) {
  if (!cfg || !out || cfg->n_in < 1 || cfg->n_in > kMlpInPad)
    return fail(WINDS_BS_ERR_ARG, "n_in must be 1..16");
  *out = nullptr;
  int nd = 0;
  if (cudaGetDeviceCount(&nd) != cudaSuccess || nd < 1) return fail(WINDS_BS_ERR_NODEV, "no CUDA device");
  winds_mlp *m = new winds_mlp();
  cudaGetDevice(&m->dev);
  m->n_in = cfg->n_in;
  cudaError_t e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, m->dev);
  if (e == cudaSuccess) e = cudaEventCreate(&m->e0);
  if (e == cudaSuccess) e = cudaEventCreate(&m->e1);
  if (e != cudaSuccess) {
    delete m;
    return cuda_fail(e, "mlp stream");
  }
  cudaStream_t s = m->stream;
  int rc;
  if ((rc = m->theta.ensure(kNParam * 4, s)) || (rc = m->theta_bf.ensure(kNParam * 2, s)) ||
      (rc = m->grad.ensure(kNParam * 4, s)) || (rc = m->mom.ensure(kNParam * 4, s)) ||
      (rc = m->vel.ensure(kNParam * 4, s)) || (rc = m->shift.ensure(64, s)) ||
      (rc = m->scale.ensure(128, s)) || (rc = m->err.ensure(16, s)) ||
      (rc = m->loss.ensure(16, s))) {
    winds_mlp_destroy(m);
    return rc;
  }
  // initial weights normal(0, 1/fan_in), biases zero, padded inputs zero
  std::vector<float> th(kNParam, 0.f);
  std::mt19937_64 gen(cfg->seed);
  for (int L = 0; L < 4; ++L) {
    const int fan = L == 0 ? cfg->n_in : W;
    std::normal_distribution<double> nd01(0.0, 1.0 / std::sqrt((double)fan));
    for (int o = 0; o < W; ++o)
      for (int i = 0; i < fan; ++i) th[mlp_off_w(L) + (long long)o * kInK[L] + i] = (float)nd01(gen);
  }
  std::normal_distribution<double> nd5(0.0, 1.0 / std::sqrt((double)W));
  for (int j = 0; j < W; ++j) th[kMlpOffW5 + j] = (float)nd5(gen);
  for (int i = 0; i < 16; ++i) m->h_shift[i] = 0.f, m->h_scale[i] = 1.f;
  e = upload(m->theta.p, th.data(), kNParam * 4, s);
  if (e == cudaSuccess) e = upload(m->shift.p, m->h_shift, 64, s);
  if (e == cudaSuccess) e = upload(m->scale.p, m->h_scale, 64, s);
  if (e == cudaSuccess) e = upload(P<float>(m->scale) + 16, &m->out_scale, 4, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(P<float>(m->scale) + 17, 0, 4, s);  // base 0
  if (e == cudaSuccess) e = cudaMemsetAsync(m->mom.p, 0, kNParam * 4, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(m->vel.p, 0, kNParam * 4, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(m->err.p, 0, 16, s);
  if (e == cudaSuccess) e = launch_mlp_to_bf16(P<float>(m->theta), P<__nv_bfloat16>(m->theta_bf), kNParam, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    winds_mlp_destroy(m);
    return cuda_fail(e, "mlp init");
  }
  *out = m;
  return WINDS_BS_OK;
}

long long winds_mlp_param_count(const winds_mlp *m) { return m ? kNParam : 0; }

int winds_mlp_get_params(winds_mlp *m, float *theta) {
  if (!m || !theta) return fail(WINDS_BS_ERR_ARG, "null argument");
  cudaSetDevice(m->dev);
  cudaStreamSynchronize(m->stream);
  cudaError_t e = cudaMemcpy(theta, m->theta.p, kNParam * 4, cudaMemcpyDeviceToHost);
  return e == cudaSuccess ? WINDS_BS_OK : cuda_fail(e, "mlp params");
}

int winds_mlp_set_params(winds_mlp *m, const float *theta) {
  if (!m || !theta) return fail(WINDS_BS_ERR_ARG, "null argument");
  cudaSetDevice(m->dev);
  cudaStreamSynchronize(m->stream);
  std::vector<float> th(theta, theta + kNParam);
  for (int o = 0; o < W; ++o)  // padded inputs of layer 1 stay zero
    for (int i = m->n_in; i < kMlpInPad; ++i) th[mlp_off_w(0) + (long long)o * kMlpInPad + i] = 0.f;
  cudaError_t e = upload(m->theta.p, th.data(), kNParam * 4, m->stream);
  if (e == cudaSuccess)
    e = launch_mlp_to_bf16(P<float>(m->theta), P<__nv_bfloat16>(m->theta_bf), kNParam, m->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(m->mom.p, 0, kNParam * 4, m->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(m->vel.p, 0, kNParam * 4, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  m->adam_t = 0;
  return e == cudaSuccess ? WINDS_BS_OK : cuda_fail(e, "mlp params");
}

int winds_mlp_set_scaling(winds_mlp *m, const float *shift, const float *scale, float out_scale) {
  if (!m || !shift || !scale || !std::isfinite(out_scale))
    return fail(WINDS_BS_ERR_ARG, "bad scaling");
  cudaSetDevice(m->dev);
  for (int i = 0; i < 16; ++i) {
    m->h_shift[i] = i < m->n_in ? shift[i] : 0.f;
    m->h_scale[i] = i < m->n_in ? scale[i] : 1.f;
  }
  m->out_scale = out_scale;
  cudaStreamSynchronize(m->stream);
  cudaError_t e = upload(m->shift.p, m->h_shift, 64, m->stream);
  if (e == cudaSuccess) e = upload(m->scale.p, m->h_scale, 64, m->stream);
  if (e == cudaSuccess) e = upload(P<float>(m->scale) + 16, &out_scale, 4, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  return e == cudaSuccess ? WINDS_BS_OK : cuda_fail(e, "mlp scaling");
}

int winds_mlp_set_base(winds_mlp *m, int base) {
  if (!m || (base != WINDS_MLP_BASE_PREVIOUS && base != WINDS_MLP_BASE_EXTRAPOLATED))
    return fail(WINDS_BS_ERR_ARG, "bad start-value base %d", base);
  cudaSetDevice(m->dev);
  cudaStreamSynchronize(m->stream);
  const float f = (float)base;
  cudaError_t e = upload(P<float>(m->scale) + 17, &f, 4, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  if (e != cudaSuccess) return cuda_fail(e, "mlp base");
  m->base = base;
  return WINDS_BS_OK;
}

int winds_mlp_get_base(const winds_mlp *m) { return m ? m->base : -1; }

int winds_mlp_get_scaling(winds_mlp *m, float *shift, float *scale, float *out_scale) {
  if (!m) return fail(WINDS_BS_ERR_ARG, "null model");
  for (int i = 0; i < m->n_in; ++i) {
    if (shift) shift[i] = m->h_shift[i];
    if (scale) scale[i] = m->h_scale[i];
  }
  if (out_scale) *out_scale = m->out_scale;
  return WINDS_BS_OK;
}

int winds_mlp_forward_host(winds_mlp *m, const float *x, long long n, float *y) {
  if (!m || n < 0 || (n > 0 && (!x || !y))) return fail(WINDS_BS_ERR_ARG, "bad arguments");
  if (n == 0) return WINDS_BS_OK;
  cudaSetDevice(m->dev);
  cudaStream_t s = m->stream;
  // rows go up in pieces (the staging of one is read beside the network on the one
  // before; its copy follows that on the stream), results come back together, up to
  // 4M rows at a time
  const long long chunk = 1 << 15, most = 1 << 22;
  StageLease stage;
  int rc;
  if ((rc = m->w.ensure(std::min(n, chunk), false, s)) || (rc = m->w.y.ensure(std::min(n, most) * 4, s)))
    return rc;
  for (long long y0 = 0; y0 < n; y0 += most) {
    const long long ny = std::min(most, n - y0);
    for (long long r0 = 0; r0 < ny; r0 += chunk) {
      const long long k = std::min(chunk, ny - r0);
      const HostSpan in = {const_cast<float *>(x + (y0 + r0) * m->n_in), m->w.xraw.p,
                           (size_t)k * m->n_in * sizeof(float)};
      const cudaError_t e = stage.upload(&in, 1, s);
      if (e != cudaSuccess) return cuda_fail(e, "mlp input upload");
      if ((rc = mlp_forward(m, P<float>(m->w.xraw), k, P<float>(m->w.y) + r0, s))) return rc;
    }
    const HostSpan out = {y + y0, m->w.y.p, (size_t)ny * 4};
    const cudaError_t e = stage.download(&out, 1, s);
    if (e != cudaSuccess) return cuda_fail(e, "mlp forward");
  }
  return check_err(m);
}

int winds_mlp_loss_grad_host(winds_mlp *m, const float *x, const float *t, long long n,
                             double *loss, float *grad) {
  if (!m || n < 1 || !x || !t) return fail(WINDS_BS_ERR_ARG, "bad arguments");
  cudaSetDevice(m->dev);
  cudaStream_t s = m->stream;
  int rc = m->w.ensure(n, true, s);
  if (!rc) rc = upload_inputs(m, x, n, s);
  if (rc) return rc;
  cudaError_t e = upload(m->w.t.p, t, n * 4, s);
  if (e != cudaSuccess) return cuda_fail(e, "mlp targets");
  MlpUpdateArgs u;
  if ((rc = gradient(m, P<float>(m->w.xraw), P<float>(m->w.t), nullptr, n, P<float>(m->loss), &u, s)))
    return rc;
  u.grad = P<float>(m->grad);
  float l = 0.f;
  e = launch_mlp_update(u, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&l, m->loss.p, 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && grad)
    e = cudaMemcpyAsync(grad, m->grad.p, kNParam * 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "mlp gradient read");
  if (loss) *loss = l;
  return check_err(m);
}

int winds_mlp_train_host(winds_mlp *m, const float *x, const float *t, long long n,
                         const winds_mlp_train_params *p, float *epoch_loss) {
  if (!m || !p || n < 1 || !x || !t || p->epochs < 0 || p->batch < 1 || !(p->lr > 0))
    return fail(WINDS_BS_ERR_ARG, "bad training arguments");
  cudaSetDevice(m->dev);
  cudaStream_t s = m->stream;
  const long long B = p->batch < n ? p->batch : n;
  const long long nbatch = cdiv(n, B);
  int rc;
  if ((rc = m->Xall.ensure(n * m->n_in * 4, s)) || (rc = m->Tall.ensure(n * 4, s)) ||
      (rc = m->idx.ensure(n * 4, s)) || (rc = m->lossbuf.ensure(nbatch * 4, s)) ||
      (rc = m->w.ensure_parts(B, s)))
    return rc;
  StageLease stage;
  const HostSpan in[] = {{const_cast<float *>(x), m->Xall.p, (size_t)n * m->n_in * 4},
                         {const_cast<float *>(t), m->Tall.p, (size_t)n * 4}};
  cudaError_t e = stage.upload(in, 2, s);
  if (e != cudaSuccess) return cuda_fail(e, "mlp training upload");
  std::vector<int> perm(n);
  for (long long i = 0; i < n; ++i) perm[i] = (int)i;
  std::mt19937_64 gen(p->seed);
  std::vector<float> bl(nbatch);
  m->train_steps = 0;
  float total_ms = 0.f;
  for (int ep = 0; ep < p->epochs; ++ep) {
    std::shuffle(perm.begin(), perm.end(), gen);
    e = upload(m->idx.p, perm.data(), n * 4, s);
    if (e != cudaSuccess) return cuda_fail(e, "mlp shuffle upload");
    cudaEventRecord(m->e0, s);
    for (long long b = 0; b < nbatch; ++b) {
      const long long r0 = b * B, nb = n - r0 < B ? n - r0 : B;
      MlpUpdateArgs u;
      if ((rc = gradient(m, P<float>(m->Xall), P<float>(m->Tall), P<int>(m->idx) + r0, nb,
                         P<float>(m->lossbuf) + b, &u, s)) ||
          (rc = adam_step(m, *p, u, s)))
        return rc;
      ++m->train_steps;
    }
    cudaEventRecord(m->e1, s);
    e = cudaMemcpyAsync(bl.data(), m->lossbuf.p, nbatch * 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(e, "mlp epoch");
    float ms = 0.f;
    cudaEventElapsedTime(&ms, m->e0, m->e1);
    total_ms += ms;
    if (epoch_loss) {
      double acc = 0.0;
      for (long long b = 0; b < nbatch; ++b) {
        const long long nb = n - b * B < B ? n - b * B : B;
        acc += (double)bl[b] * (double)nb;
      }
      epoch_loss[ep] = (float)(acc / (double)n);
    }
    if ((rc = check_err(m))) return rc;
  }
  m->train_ms = total_ms;
  return WINDS_BS_OK;
}

int winds_mlp_train_stats(winds_mlp *m, double *ms, long long *steps) {
  if (!m) return fail(WINDS_BS_ERR_ARG, "null model");
  if (ms) *ms = m->train_ms;
  if (steps) *steps = m->train_steps;
  return WINDS_BS_OK;
}

void winds_mlp_destroy(winds_mlp *m) {
  if (!m) return;
  cudaSetDevice(m->dev);
  if (m->stream) cudaStreamSynchronize(m->stream);
  m->w.release();
  for (DevBuf *b : {&m->theta, &m->theta_bf, &m->grad, &m->mom, &m->vel, &m->shift, &m->scale,
                    &m->err, &m->loss, &m->lossbuf, &m->idx, &m->Xall, &m->Tall})
    b->release();
  if (m->e0) cudaEventDestroy(m->e0);
  if (m->e1) cudaEventDestroy(m->e1);
  if (m->stream) cudaStreamDestroy(m->stream);
  delete m;
}

}  // extern "C"
