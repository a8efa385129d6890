// host_stage.h -- transfers between pageable host arrays and the device through
// pinned staging memory.
//
// The driver stages a pageable copy by itself, array by array on the calling thread.
// Here up to 1 MB of inputs goes up in one DMA per run of device memory (two
// evaluations on 3.1k host points 400 us instead of 490); larger inputs are left to the
// driver, which is as fast (4.4 MB: 290 us; through here with two to eight threads 500).
//
// Outputs come back in DMAs of 1 MB, each copied out while the next are under way. The
// calling thread does so alone up to 8 MB, with another up to 16 MB; beyond, the driver
// copies into pages that are there and eight threads make those that are not. Host
// evaluations (of little else) by the size of their output, in us, into an array just
// allocated and into one in use:
//                     1.4 MB      4.6 MB       11 MB        23 MB        34 MB
//   the driver      507   371  1237   739  2450  1552  4516   2824  10880   4216
//   one thread      428   388   992   846  2213  1873  5371   4266   9967   7723
//   two             690   630  1118   930  2020  1618  4325   3354   8336   5901
//   one per MB      417   383  1517  1029  3261  1758  5195   3173   6243   5762
// and a wake's state of 6.7 MB 1170, 820, 770 and 1610 us. Kinematics, with threads that
// start next to the last kernel, take one per MB, up to eight (28 MB: 0.9 to 1.2 ms, the
// driver 1.98, one thread 2.60).
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
// from a pool that keeps at most kKept of them per device, each of at most kMaxPinned
// bytes (and the quarter that HostBuf adds, 40 MB) and kMaxDev; the others are freed when they come back. Any
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
  // Copies the spans after the work on s; returns when all are written. wide: with a
  // thread per MB, up to eight, whatever the pages.
  cudaError_t download(const HostSpan *v, int n, cudaStream_t s, bool wide = false);

  struct Stage;

 private:
  Stage *st_ = nullptr;
  cudaError_t err_ = cudaSuccess;
};

void release_stages();  // the pool's memory (no lease may be held)

}  // namespace winds
