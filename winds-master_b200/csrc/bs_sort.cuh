// bs_sort.cuh -- targets of one group sorted along a Hilbert curve by one CTA:
// bounding box, keys, radix sort and gather in a single launch. For groups of
// up to kBlockSortMax targets; larger ones take the device-wide radix sort
// (launch_sort_targets). On 3.1k targets one launch of 31 us takes the place of
// 13, whose eight passes over 64-bit keys alone took 72 us.
#pragma once

#include <cub/block/block_radix_sort.cuh>

#include "bs_device.cuh"

namespace winds {

constexpr int kSortThreads = 1024;
constexpr int kSortBits = 5;   // radix digit: 25-bit keys take five passes
constexpr int kKeyBits = 25;   // 8 bits a coordinate, and bit 24: the target is unused

// Spreads the low 10 bits of v so that they occupy every third bit.
__device__ __forceinline__ unsigned spread3(unsigned v) {
  unsigned x = v & 0x3ffu;
  x = (x | (x << 16)) & 0x30000ffu;
  x = (x | (x << 8)) & 0x300f00fu;
  x = (x | (x << 4)) & 0x30c30c3u;
  x = (x | (x << 2)) & 0x9249249u;
  return x;
}

// Distance along a 3-D Hilbert curve of 10 bits a coordinate (Skilling's
// transpose algorithm, "Programming the Hilbert curve", AIP Conf. Proc. 707,
// 2004); its leading bits are the distance at a coarser resolution. Consecutive
// targets on it are neighbours in space without exception, where a Morton code
// jumps at every power of two: on the large wake the radius of 96 consecutive
// targets is 9.1 m (median; largest 34 m) instead of 10.1 m (82 m).
__device__ __forceinline__ unsigned hilbert30(unsigned x, unsigned y, unsigned z) {
  unsigned X[3] = {x, y, z};
#pragma unroll
  for (unsigned Q = 512u; Q > 1u; Q >>= 1) {
    const unsigned m = Q - 1u;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (X[c] & Q) {
        X[0] ^= m;
      } else {
        const unsigned t = (X[0] ^ X[c]) & m;
        X[0] ^= t;
        X[c] ^= t;
      }
    }
  }
  X[1] ^= X[0];
  X[2] ^= X[1];
  unsigned t = 0;
#pragma unroll
  for (unsigned Q = 512u; Q > 1u; Q >>= 1)
    if (X[2] & Q) t ^= Q - 1u;
  return spread3(X[0] ^ t) << 2 | spread3(X[1] ^ t) << 1 | spread3(X[2] ^ t);
}

// The Hilbert position of p in the box [lo, hi] (floats).
__device__ __forceinline__ unsigned hilbert_key(const double p[3], const float lo[3],
                                                const float hi[3]) {
  unsigned cell[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double w = hi[c] > lo[c] ? (double)hi[c] - (double)lo[c] : 1.0;
    double u = (p[c] - (double)lo[c]) / w * 1023.999;
    if (!(u >= 0.0)) u = 0.0;  // also catches NaN
    if (u > 1023.0) u = 1023.0;
    cell[c] = (unsigned)u;
  }
  return hilbert30(cell[0], cell[1], cell[2]);
}

// Targets of a MATLAB array P [ns, 3, ...]; one group.
struct MatlabTargets {
  const double *P;
  long long ns;
  int n;
  __device__ int count(int) const { return n; }
  __device__ long long offset(int) const { return 0; }
  __device__ bool load(int, int t, double p[3]) const {
    const long long j = t / ns, b = t - j * ns + ns * 3 * j;
    p[0] = P[b], p[1] = P[b + ns], p[2] = P[b + 2 * ns];
    return true;
  }
};

template <int ITEMS>
using TargetSort = cub::BlockRadixSort<unsigned, kSortThreads, ITEMS, int, kSortBits>;

// One CTA per group of SRC. tp: the sorted targets (w = 1 and the origin for
// unused ones, which come last); perm: their places in the input order.
template <int ITEMS, class SRC>
__global__ void __launch_bounds__(kSortThreads) bs_sort_targets(const SRC src, double4 *tp,
                                                                int *perm, BBox *bb) {
  extern __shared__ __align__(16) unsigned char sort_smem[];
  auto &temp = *reinterpret_cast<typename TargetSort<ITEMS>::TempStorage *>(sort_smem);
  __shared__ float s_lo[3][32], s_hi[3][32];
  const int g = blockIdx.x, n = src.count(g), tid = threadIdx.x;
  const long long off = src.offset(g);
  float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  for (int t = tid; t < n; t += kSortThreads) {
    double p[3];
    if (src.load(g, t, p))
#pragma unroll
      for (int c = 0; c < 3; ++c) lo[c] = fminf(lo[c], (float)p[c]), hi[c] = fmaxf(hi[c], (float)p[c]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
      hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
    }
    if ((tid & 31) == 0) s_lo[c][tid >> 5] = lo[c], s_hi[c][tid >> 5] = hi[c];
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    lo[c] = s_lo[c][tid & 31], hi[c] = s_hi[c][tid & 31];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
      hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
    }
    if (tid == c && lo[c] != FLT_MAX) atomicMin(&bb->tmin[c], float_key(lo[c]));
    if (tid == c && hi[c] != -FLT_MAX) atomicMax(&bb->tmax[c], float_key(hi[c]));
  }
  unsigned key[ITEMS];
  int val[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int t = tid * ITEMS + k;
    val[k] = t;
    key[k] = (1u << kKeyBits) - 1u;  // past the end: after the last target, as the sort is stable
    if (t < n) {
      double p[3];
      const bool used = src.load(g, t, p);
      key[k] = used ? hilbert_key(p, lo, hi) >> 6 : 1u << (kKeyBits - 1);
    }
  }
  TargetSort<ITEMS>(temp).SortBlockedToStriped(key, val, 0, kKeyBits);
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int r = k * kSortThreads + tid;
    if (r < n) {
      double p[3];
      const bool used = src.load(g, val[k], p);
      tp[off + r] = used ? make_double4(p[0], p[1], p[2], 0.0) : make_double4(0.0, 0.0, 0.0, 1.0);
      perm[off + r] = (int)(off + val[k]);
    }
  }
}

template <int ITEMS, class SRC>
cudaError_t launch_block_sort_t(const SRC &src, int groups, double4 *tp, int *perm, BBox *bb,
                                cudaStream_t s) {
  const int smem = (int)sizeof(typename TargetSort<ITEMS>::TempStorage);
  cudaError_t e = cudaFuncSetAttribute(bs_sort_targets<ITEMS, SRC>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  bs_sort_targets<ITEMS, SRC><<<groups, kSortThreads, smem, s>>>(src, tp, perm, bb);
  return cudaGetLastError();
}

// max_n: the largest group, at most kBlockSortMax.
template <class SRC>
cudaError_t launch_block_sort(const SRC &src, int groups, long long max_n, double4 *tp, int *perm,
                              BBox *bb, cudaStream_t s) {
  if (max_n <= 2 * kSortThreads) return launch_block_sort_t<2>(src, groups, tp, perm, bb, s);
  if (max_n <= 4 * kSortThreads) return launch_block_sort_t<4>(src, groups, tp, perm, bb, s);
  if (max_n <= 8 * kSortThreads) return launch_block_sort_t<8>(src, groups, tp, perm, bb, s);
  return launch_block_sort_t<16>(src, groups, tp, perm, bb, s);
}

}  // namespace winds
