// A CUDA runtime of a few calls for the host transfers (csrc/host_stage.cu) on a machine without a GPU:
// "device" memory is host memory, copies are done at once, an event's wait takes as long as the test says,
// and the test makes calls fail.
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <thread>

#include "host_stage.h"

static int g_wait_ms = 0;
static int g_fail_pinned = 0;
static int g_copies = 0;
static cudaError_t g_last = cudaSuccess;

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
  std::this_thread::sleep_for(std::chrono::milliseconds(g_wait_ms));
  g_wait_ms = 0;  // the first of a transfer waits for the work before it
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  ++g_copies;
  return cudaSuccess;
}

// Device bytes to host through one lease, after work of `wait_ms`; pinned memory not to be had if fail_pinned.
int stage_download(void *host, void *dev, size_t bytes, int wait_ms, int fail_pinned,
                   int wide) {
  g_wait_ms = wait_ms, g_fail_pinned = fail_pinned, g_copies = 0;
  winds::StageLease stage;
  const winds::HostSpan v = {host, dev, bytes};
  return (int)stage.download(&v, 1, (cudaStream_t)1, wide != 0);
}
int stage_upload(void *host, void *dev, size_t bytes, int fail_pinned) {
  g_fail_pinned = fail_pinned;
  winds::StageLease stage;
  const winds::HostSpan v = {host, dev, bytes};
  return (int)stage.upload(&v, 1, (cudaStream_t)1);
}
int stage_copies(void) { return g_copies; }
int stage_last_error(void) { return (int)cudaGetLastError(); }
void stage_release(void) { winds::release_stages(); }
}

namespace winds {
int HostBuf::ensure(size_t bytes) {
  if (bytes <= cap) return 0;
  release();
  if (g_fail_pinned) {
    g_last = cudaErrorMemoryAllocation;
    return 4;
  }
  p = std::malloc(bytes);
  cap = bytes;
  return 0;
}
void HostBuf::release() { std::free(p); p = nullptr; cap = 0; }
int DevBuf::ensure(size_t, cudaStream_t) { return 0; }
void DevBuf::release() {}
}  // namespace winds
