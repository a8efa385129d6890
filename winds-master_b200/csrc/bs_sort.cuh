// bs_sort.cuh -- targets of each group ordered along a Hilbert curve by counting:
// a target's place is the number of keys below its own.
#pragma once

#include "bs_device.cuh"
#include "bs_launch.h"

namespace winds {

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

// The one group of an evaluation's targets.
struct OneGroup {
  int n;
  __device__ int count(int) const { return n; }
  __device__ long long offset(int) const { return 0; }
};

// A block places 32 R targets of a group, R a lane; each of its warps counts a run
// of the group's keys, read by the warp into shared memory and from there four at a
// time. Keys are whole numbers below 2^24 as floats, so that a key and one more are
// exact (2^24 + 1 is no float) and a comparison is a saturated difference, at the full rate of the FP32 units where an integer
// comparison has half: 16k targets take 28 us (as integers 41), 3.2k 6
// (11.4). R: enough blocks for the SMs before fewer reads of the keys.
constexpr int kRankWarps = 16;
constexpr float kUnusedKey = 16777215.f;  // after every live target's
template <int R, class GROUPS>
__global__ void __launch_bounds__(32 * kRankWarps)
    bs_rank_targets(const GROUPS gr, const float *__restrict__ keys,
                    const double4 *__restrict__ tp_raw, double4 *tp, int *perm) {
  after_previous();
  extern __shared__ float4 s_key[];  // a run of `run` keys per warp
  __shared__ float s_cnt[kRankWarps][32 * R];
  const int g = blockIdx.y, n = gr.count(g), i0 = blockIdx.x * 32 * R;
  if (i0 >= n) return;
  const long long off = gr.offset(g);
  const float *key = keys + off;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int run = ((n + kRankWarps - 1) / kRankWarps + 3) / 4, j0 = 4 * run * warp;  // run: of four
  const float inf = __int_as_float(0x7f800000);
  float *mine = reinterpret_cast<float *>(s_key + run * warp);
  for (int j = lane; j < 4 * run; j += 32) mine[j] = j0 + j < n ? key[j0 + j] : inf;
  float k[R], c[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int i = i0 + 32 * q + lane;
    k[q] = i < n ? key[i] : 0.f;
    c[q] = 0.f;
  }
  __syncwarp();
  // keys before the block come first where equal, those after it do not
  const float4 *x = s_key + run * warp;
  const int lo = min(max((i0 - j0) / 4, 0), run), hi = min(max((i0 - j0) / 4 + 8 * R, 0), run);
  const auto count = [&](int f, int t, float add) {
#pragma unroll 4
    for (int j = f; j < t; ++j) {
      const float4 v = x[j];
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const float y = k[q] + add;
        c[q] += (__saturatef(y - v.x) + __saturatef(y - v.y)) +
                (__saturatef(y - v.z) + __saturatef(y - v.w));
      }
    }
  };
  count(0, lo, 1.f);
  count(hi, run, 0.f);
  for (int j = lo; j < hi; ++j) {
    const float4 v = x[j];
    const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < R; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        c[q] += __saturatef(k[q] + (j0 + 4 * j + e < i0 + 32 * q + lane ? 1.f : 0.f) - w[e]);
  }
#pragma unroll
  for (int q = 0; q < R; ++q) s_cnt[warp][32 * q + lane] = c[q];
  __syncthreads();
  const int i = i0 + (int)threadIdx.x;
  if (threadIdx.x >= 32 * R || i >= n) return;
  float r = 0.f;
#pragma unroll
  for (int w = 0; w < kRankWarps; ++w) r += s_cnt[w][threadIdx.x];
  tp[off + (int)r] = tp_raw[off + i];
  perm[off + (int)r] = (int)(off + i);
}

// Shared memory of a block for groups of up to n targets.
constexpr int rank_smem(long long n) {
  return ((int)((n + kRankWarps - 1) / kRankWarps) + 3) / 4 * kRankWarps * (int)sizeof(float4);
}

template <int R, class GROUPS>
cudaError_t launch_rank_targets(const GROUPS &gr, int groups, long long max_n, const TargetBufs &b,
                                cudaStream_t s) {
  // The attribute is the function's, for all threads: always the largest group's size, so
  // that no call can set less between another's setting and its launch.
  const cudaError_t e =
      cudaFuncSetAttribute(bs_rank_targets<R, GROUPS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           rank_smem(kCountingTargets));
  if (e != cudaSuccess) return e;
  const int smem = rank_smem(max_n);
  const dim3 grid((unsigned)((max_n + 32 * R - 1) / (32 * R)), (unsigned)groups);
  launch_after(bs_rank_targets<R, GROUPS>, grid, 32 * kRankWarps, smem, s, gr,
               reinterpret_cast<const float *>(b.keys), b.tp_raw, b.tp, b.perm);
  return cudaGetLastError();
}

// n targets in tp_raw (tgroup: their groups; not read by the counting sort).
template <class GROUPS>
cudaError_t launch_order_targets(const GROUPS &gr, int groups, long long max_n, long long n,
                                 const TargetBufs &b, const BBox *bb, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (!sort_by_counting(groups, max_n)) return launch_sort_targets(b, n, groups, bb, s);
  const cudaError_t e = launch_target_keys(b.tp_raw, n, bb, reinterpret_cast<float *>(b.keys), s);
  if (e != cudaSuccess) return e;
  const long long warps = groups * ((max_n + 31) / 32);
  if (warps <= 148) return launch_rank_targets<1>(gr, groups, max_n, b, s);
  if (warps <= 2 * 148) return launch_rank_targets<2>(gr, groups, max_n, b, s);
  return launch_rank_targets<4>(gr, groups, max_n, b, s);
}

}  // namespace winds
