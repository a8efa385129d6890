// bs_launch.h -- host-side launchers of the induced-velocity kernels.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "bs_types.h"
#include "winds_bs.h"

namespace winds {

// Launches a kernel that begins with after_previous() so that its blocks may be set
// up while the kernel before it in the stream still runs: an evaluation's seven
// launches on 3.1k targets take 117 us instead of 126. Not for the direct sums, whose
// workers are as many per SM: set up beside blocks of the kernel before they are
// spread unevenly (7.6k targets 404 us instead of 325).
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                         A &&...args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}


struct PackedFilaments {
  float4 *pk;  // records: 4 float4 per filament (layout in bs_types.h)
  double4 *ra, *rb;
};

// Filament ranges of groups are multiples of this (a multiple of every FP32 tile
// size and of the FP64 stage).
constexpr int kFilamentPad = 128;

bool f32c_config_supported(int T, int KF);
// FP32c work runs on independent warp workers: a tile holds f32c_tile(T)
// targets, f32c_occupancy() counts resident workers per SM, and launch_f32c's
// grid counts workers.
int f32c_targets(int T);  // targets per lane that a choice of T runs with
int f32c_tile(int T);
int f32c_quantum(int KF);  // filaments of an item: a multiple of this
int f32c_warps();          // workers per CTA
int f64_threads();
int f64_tile();
int f32c_occupancy(int model, int T, int KF);
int f64_occupancy(int model, double n, bool sequential);
unsigned long long default_wait_limit_ns();

// First kernel of an evaluation: empty bounding box, work queue at its start,
// near (2 words) and cnt (2 kPackFams words) zero.
cudaError_t launch_begin(BBox *bb, unsigned *ctr, unsigned long long *near, unsigned long long *cnt,
                         cudaStream_t s);
// Targets sorted by (group, place on a Hilbert curve), from tp_raw. Counting
// needs tp, perm, tp_raw and one 32-bit key a target; the device-wide sort needs the
// rest too (keys: two words of 32 bits for one group, of 64 for more).
struct TargetBufs {
  double4 *tp, *tp_raw;
  int *tgroup, *vals, *perm;
  unsigned long long *keys;
  void *sort_tmp;
  size_t sort_bytes;
};
// Counting compares each target with its group's others: 3.2k targets take 6 us, 16k
// 28 and 22k 65, against 66 us and more launches for the device-wide sort of 31-bit
// keys; past 148 blocks of 128 targets some SMs have two. (One CTA per group with a
// radix sort in shared memory: 31 us on 3.2k, 121 on 16k.) More groups share the
// same units, so the line is their sum of squares.
constexpr long long kCountingMax = 360ll * 1000 * 1000;
constexpr long long kCountingTargets = 18973;  // most of one group
static_assert(kCountingTargets * kCountingTargets <= kCountingMax &&
                  (kCountingTargets + 1) * (kCountingTargets + 1) > kCountingMax,
              "largest group that is counted");
inline bool sort_by_counting(long long groups, long long max_n) {
  return max_n <= kCountingTargets && groups * max_n * max_n <= kCountingMax;
}
// Packs the families (device arrays) one after the other, in input order or
// (cnt: as launch_begin leaves it) each in the order with more links between
// neighbours, then inert filaments up to pad_to, and the nt targets P [ns,3,...]
// into tb.tp_raw. Adds to *launches.
cudaError_t launch_pack(const winds_bs_family *fams, int nfam, unsigned long long *cnt,
                        long long pad_to, int model, double dcut, const PackedFilaments &pf,
                        const double *P, long long ns, long long nt, const TargetBufs &tb, BBox *bb,
                        cudaStream_t s, int *launches);
cudaError_t launch_target_keys(const double4 *tp, long long n, const BBox *bb, float *keys,
                               cudaStream_t s);
// The n targets of one group in order.
cudaError_t launch_order_targets(long long n, const TargetBufs &b, const BBox *bb, cudaStream_t s);
// Device-wide sort of n targets already in tp_raw / tgroup (groups of them), and
// the scratch bytes it needs.
cudaError_t launch_sort_targets(const TargetBufs &b, long long n, int groups, const BBox *bb,
                                cudaStream_t s);
cudaError_t sort_targets_bytes(long long n, int groups, size_t *bytes);
cudaError_t launch_f32c(const F32cArgs &a, int model, int T, int KF, int grid, cudaStream_t s);
// sequential: every target's terms in the filaments' order, as ref_pair has them.
cudaError_t launch_f64(const F32cArgs &a, bool sequential, int grid, cudaStream_t s);
// live (with the plan's items): only each group's live part (GroupLive). Leaves
// the work queue's counter ctr at its start.
cudaError_t launch_reduce(const Tile *tiles, int n_tiles, const Group *groups, const double *part,
                          const int *perm, int tile_cap, unsigned *ctr, cudaStream_t s,
                          const Item *items = nullptr, const GroupLive *live = nullptr);
cudaError_t launch_ffma_peak(float *out, int blocks, int iters, cudaStream_t s);
cudaError_t launch_wait_selftest(unsigned *err, unsigned long long limit_ns, cudaStream_t s);
// y [4][n]: rsqrt64, rcp64 and CUDA's rsqrt and 1 / x of x [n].
cudaError_t launch_roots_selftest(const double *x, long long n, double *y, cudaStream_t s);
cudaError_t launch_length(const double *F1, const double *F2, long long d0, long long nf, double *L,
                          cudaStream_t s);

}  // namespace winds
