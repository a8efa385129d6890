// host_stage.h -- transfers between pageable host arrays and the device through
// pinned staging memory.
//
// The driver stages a pageable copy by itself, array by array on the calling
// thread. Here up to 1 MB of inputs goes up in one DMA per run of device memory, and
// outputs come back in DMAs of 1 MB that up to eight threads copy out while the next
// are under way: 29 MB of kinematics in 15 arrays take 0.99 ms instead of 2.84, two
// evaluations on 3.1k host points 400 us instead of 490, a step's status and state
// 100 us less. Larger inputs are left to the driver, which is as fast (4.4 MB: 290 us; through
// here with two to eight threads 500).
#pragma once

#include <cuda_runtime.h>

#include "engine.h"

namespace winds {

struct HostSpan {
  void *host;
  void *dev;
  size_t bytes;
};

// Pinned memory, a stream and device scratch for one transfer or call at a time,
// from a pool that keeps at most kKept of them per device, each of at most
// kMaxPinned and kMaxDev bytes; the others are freed when they come back. Any
// number of threads may hold one each.
class StageLease {
 public:
  static constexpr size_t kMaxPinned = 32u << 20, kMaxDev = 256u << 20;
  static constexpr int kKept = 2;
  StageLease();
  ~StageLease();
  StageLease(const StageLease &) = delete;
  StageLease &operator=(const StageLease &) = delete;
  cudaError_t error() const { return err_; }
  cudaStream_t stream() const;
  DevBuf &scratch();  // device memory, free for the lease's holder

  // Enqueues the spans on s; pageable sources are read before it returns. Host memory
  // that is not plain pageable memory is copied from (and to) directly.
  cudaError_t upload(const HostSpan *v, int n, cudaStream_t s);
  // Copies the spans after the work on s; returns when all are written.
  cudaError_t download(const HostSpan *v, int n, cudaStream_t s);

  struct Stage;

 private:
  Stage *st_ = nullptr;
  cudaError_t err_ = cudaSuccess;
};

void release_stages();  // the pool's memory (no lease may be held)

}  // namespace winds
