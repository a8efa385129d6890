// mlp_kernels.cu -- kernels of the MLP that predicts the converged bound
// circulation (the Kutta-Joukowski initial guess).
//
// mlp_net runs the whole network on a tile of 128 rows without leaving the SM,
// forward (inference) or forward and backward (training). The weights (100 KB in
// BF16) stay in shared memory, activations go from one layer's epilogue into the
// shared-memory operand of the next, pre-activations stay in tensor memory.
// GEMMs run on the 5th-generation tensor cores: operands in the no-swizzle
// core-matrix layout (8 rows x 16 bytes per core matrix), one thread issues
// tcgen05.mma (kind::f16, BF16 x BF16 -> FP32, M = 128) into a tensor-memory
// accumulator and commits to an mbarrier, and warps read the accumulator back
// with tcgen05.ld (a warp of quadrant q owns lanes 32q..32q+31, one row a thread).
//
// One shared-memory tile serves both operand majors: the tile of a row-major
// [R][C] matrix is stored with element (r, c) at
//     (r / 8) * (C / 8) * 128 + (c / 8) * 128 + (r % 8) * 16 + (c % 8) * 2   bytes,
// which is the K-major canonical layout when rows are M (or N) and columns K
// (LBO = 128 between K chunks, SBO = C/8*128 between row groups), and the
// MN-major canonical layout when rows are K and columns M (or N) (SBO = 128
// between M groups, LBO = C/8*128 between K groups). So activations stored
// [rows][features] and weights stored [out][in] feed the forward GEMM, the
// input-gradient GEMM and the weight-gradient GEMM without transposes.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "bs_device.cuh"
#include "bs_launch.h"
#include "mlp_launch.h"

namespace winds {
namespace {

constexpr int kTileM = 128;
constexpr int kNetThreads = 512;

// ------------------------------------------------------- tcgen05 wrappers
// Shared-memory matrix descriptor (no swizzle): start address, leading and
// stride byte offsets (all >> 4), descriptor version 1 at bits 46-47.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1u << 46;
  return d;
}

// Instruction descriptor, kind::f16: D FP32 (bits 4-5 = 1), A and B BF16
// (bits 7-9, 10-12 = 1), operand majors (bits 15, 16: 1 = MN-major),
// N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__device__ __forceinline__ uint32_t umma_idesc(int M, int N, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(slot)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Generic-proxy shared-memory writes made visible to the tensor cores.
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrives on `bar` once every MMA this thread issued before has completed.
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

// 32 lanes x 16 consecutive 32-bit columns: thread i gets lane (base + i).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float (&v)[16]) {
  uint32_t r[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(v[i]);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
      "%11, %12, %13, %14, %15};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Arrives on the barrier at this shared-memory address of another CTA of the cluster.
__device__ __forceinline__ void mbar_arrive_cluster(uint64_t *bar, unsigned rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(bar)), "r"(rank));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Barriers of a group of threads (id 1 and up; 0 is __syncthreads).
__device__ __forceinline__ void group_sync(int id, int threads) {
  __syncwarp();
  asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ bool group_and(int id, int threads, bool p) {
  uint32_t r;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %3, 0;\n\t"
      "barrier.cta.red.and.aligned.pred q, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(threads), "r"((uint32_t)p)
      : "memory");
  return r != 0;
}

// ----------------------------------------------------------- activation
// GELU, tanh form: 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))). (As z /
// (1 + exp(-2u)) it takes fewer instructions and is as accurate, but its last bits
// move activations across BF16 rounding boundaries: outputs 1e-4 of their size.)
constexpr float kGeluC = 0.7978845608028654f;  // sqrt(2/pi)
constexpr float kGeluA = 0.044715f;

template <bool GRAD>
__device__ __forceinline__ float gelu(float z, float *grad) {
  const float z2 = z * z;
  const float t = tanhf(kGeluC * fmaf(kGeluA * z, z2, z));
  if (GRAD) *grad = 0.5f * (1.f + t) + 0.5f * z * (1.f - t * t) * kGeluC * fmaf(3.f * kGeluA, z2, 1.f);
  return 0.5f * z * (1.f + t);
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&h);
}

// Bytes from the start of a [128][128] tile to columns [8 c8, 8 c8 + 8) of row r.
__device__ __forceinline__ int tile_offset(int r, int c8) {
  return (r >> 3) * 2048 + c8 * 128 + (r & 7) * 16;
}

// ---------------------------------------------------------------- mlp_net
constexpr int kTileBytes = kTileM * kMlpWidth * 2;   // 32 KB
constexpr int kSmallTileBytes = kTileM * kMlpInPad * 2;

template <bool TRAIN>
struct NetSmem {
  static constexpr int G = TRAIN ? 1 : 2;  // groups of threads, a tile each
  unsigned char w1[kSmallTileBytes];
  unsigned char w[3][kTileBytes];
  unsigned char x[G][kSmallTileBytes];
  unsigned char a[TRAIN ? 3 : G][kTileBytes];  // activations: of each layer, of each group
  float bias[4][kMlpWidth];
  float w5[kMlpWidth];
  float shift[kMlpInPad], scale[kMlpInPad];
  float colsum[TRAIN ? 4 : 1][kMlpWidth];
  float dy[TRAIN ? kTileM : 1], e[TRAIN ? kTileM : 1];
  uint64_t mbar[G], chain[3];
  uint32_t tmem_slot;
};
static_assert(sizeof(NetSmem<true>) <= 227 * 1024, "training tile");
// More than half an SM's shared memory: one CTA per SM, whose tensor memory the
// allocation below never has to wait for.
static_assert(sizeof(NetSmem<false>) > 114 * 1024, "one CTA per SM");

// D = A B (or D += A B) of one tile, issued by one thread: A [128 x 16 steps]
// and B in tiles of `ca` and `cb` columns, K- or MN-major.
__device__ __forceinline__ void tile_mma(uint32_t d, uint32_t a, int a_mn, int ca, uint32_t b, int b_mn,
                                         int cb, int n, int steps, int add) {
  const uint32_t idesc = umma_idesc(kTileM, n, a_mn, b_mn);
  const uint32_t ga = (ca / 8) * 128, gb = (cb / 8) * 128;  // between groups of 8 rows
  for (int j = 0; j < steps; ++j)
    tc_mma(d, umma_desc(a + j * (a_mn ? 2 * ga : 256u), a_mn ? ga : 128u, a_mn ? 128u : ga),
           umma_desc(b + j * (b_mn ? 2 * gb : 256u), b_mn ? gb : 128u, b_mn ? 128u : gb), idesc,
           j > 0 || add ? 1u : 0u);
}

// Row-major [128][C] weights into a tile, asynchronously; eight threads with
// consecutive rows fill one core matrix (no bank conflicts).
template <int C>
__device__ __forceinline__ void load_weights(unsigned char *dst, const __nv_bfloat16 *src) {
#pragma unroll
  for (int v = threadIdx.x; v < 128 * (C / 8); v += kNetThreads) {
    const int r = (v / C) * 8 + (v & 7), c8 = (v >> 3) % (C / 8);
    cp_async16(dst + (r >> 3) * (C / 8) * 128 + c8 * 128 + (r & 7) * 16, src + r * C + 8 * c8);
  }
}

// Sum over a warp's lanes of 32 columns; lane l returns column l's.
__device__ __forceinline__ float column_sums(float (&v)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

// Bound by the epilogues' tanh: 16k elements a tile and layer at some 60
// instructions, against 128 cycles of MMA. One CTA per SM (the weights fill its
// shared memory). Inference: two groups of 256 threads with a tile each, so that
// the epilogue of one covers the MMA and the barriers of the other. Training: 512
// threads on one tile, whose gelu' of three layers and accumulators take all 512
// columns of tensor memory. As one launch per GEMM, with activations through
// memory, 100k rows forward took 236 us of device time and a step on 4096 rows
// 349 us; now 97 and 54 us (73 with the weight gradients' parts row by row).
template <bool TRAIN>
__global__ void __launch_bounds__(kNetThreads, 1) mlp_net(const MlpNetArgs g) {
  after_previous();
  extern __shared__ __align__(1024) unsigned char net_smem[];
  using Smem = NetSmem<TRAIN>;
  Smem &sm = *reinterpret_cast<Smem *>(net_smem);
  constexpr int G = Smem::G;
  constexpr int GT = kNetThreads / G;    // threads of a group
  constexpr int CPT = 128 / (GT / 128);  // columns of a thread: 32 or 64
  constexpr uint32_t kCols = TRAIN ? 512 : 256;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int grp = tid / GT, gt = tid % GT, bar = 1 + grp;
  const int quad = warp & 3, colg = gt >> 7, c0 = colg * CPT;
  const int rank = blockIdx.x & 1;  // in the pair (training)
  const int row = quad * 32 + lane;  // of the tile: this thread's tensor-memory lane
  if (warp == 0) tmem_alloc(&sm.tmem_slot, kCols);
  if (tid == 0) {
    for (int k = 0; k < G; ++k) mbar_init(&sm.mbar[k], 1);
    for (int k = 0; k < 3; ++k) mbar_init(&sm.chain[k], 1);
    fence_mbar_init();
  }
  load_weights<kMlpInPad>(sm.w1, g.wbf + mlp_off_w(0));
#pragma unroll
  for (int L = 1; L < 4; ++L) load_weights<kMlpWidth>(sm.w[L - 1], g.wbf + mlp_off_w(L));
  for (int i = tid; i < 4 * kMlpWidth; i += kNetThreads)
    sm.bias[i >> 7][i & 127] = g.theta[mlp_off_b(i >> 7) + (i & 127)];
  if (tid < kMlpWidth) sm.w5[tid] = g.theta[kMlpOffW5 + tid];
  if (tid < kMlpInPad) {
    sm.shift[tid] = tid < g.n_in ? g.shift[tid] : 0.f;
    sm.scale[tid] = tid < g.n_in ? g.scale[tid] : 0.f;
  }
  const float b5 = g.theta[kMlpOffB5];
  cp_async_wait_all();
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  if constexpr (TRAIN) cooperative_groups::this_cluster().sync();  // both CTAs' barriers are set up
  tc_fence_after();
  const uint32_t tmem = sm.tmem_slot + (TRAIN ? 0u : 128u * grp);
  const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
  uint64_t *mbar = &sm.mbar[grp];
  uint32_t phase = 0;
  bool ok = true;
  const uint32_t s_x = smem_u32(sm.x[grp]), s_w1 = smem_u32(sm.w1);
  const auto s_a = [&](int L) { return smem_u32(sm.a[TRAIN ? L : grp]); };
  const auto s_w = [&](int L) { return smem_u32(sm.w[L - 1]); };
  // operands written by all threads of the group, then one thread's MMAs
  const auto ready = [&] {
    fence_async_smem();
    tc_fence_before();
    group_sync(bar, GT);
    if (gt == 0) tc_fence_after();
  };
  const auto wait = [&] {
    const bool done = mbar_wait_bounded(mbar, phase, g.err, g.wait_limit_ns);
    phase ^= 1u;
    ok = group_and(bar, GT, done);
    tc_fence_after();
    return ok;
  };
  const long long tiles = (g.n + kTileM - 1) / kTileM;
  for (long long tile = blockIdx.x + (long long)grp * gridDim.x; tile < tiles && ok;
       tile += (long long)G * gridDim.x) {
    const long long r0 = tile * kTileM;
    const bool valid = r0 + row < g.n;
    // inputs: standardised, padded with zeros, as BF16
    if (gt < 2 * kTileM) {
      const int r = gt >> 1, h = gt & 1;
      uint32_t p[4] = {0u, 0u, 0u, 0u};
      if (r0 + r < g.n) {
        const long long src = g.idx ? g.idx[r0 + r] : r0 + r;
        const float *x = g.x + src * g.n_in;
        float v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int k = 8 * h + c;
          v[c] = k < g.n_in ? (x[k] - sm.shift[k]) * sm.scale[k] : 0.f;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) p[q] = pack_bf16(v[2 * q], v[2 * q + 1]);
      }
      *reinterpret_cast<uint4 *>(sm.x[grp] + (r >> 3) * 256 + h * 128 + (r & 7) * 16) =
          make_uint4(p[0], p[1], p[2], p[3]);
    }
    float t = 0.f;
    if (TRAIN && valid) t = g.t[g.idx ? g.idx[r0 + row] : r0 + row];
    // ---- forward: z_L = a_{L-1} W_L^T + b_L, a_L = gelu(z_L)
    float yp[CPT / 4];               // output layer: sums of four columns
    float gp[TRAIN ? 32 : 1];        // layer 4 (training): gelu'
    uint32_t a4[TRAIN ? 16 : 1];     // and activations
#pragma unroll 1
    for (int L = 0; L < 4; ++L) {
      const uint32_t acc = tmem + (TRAIN ? 128u * L : 0u);
      ready();
      if (gt == 0) {
        if (L == 0)
          tile_mma(acc, s_x, 0, kMlpInPad, s_w1, 0, kMlpInPad, kMlpWidth, 1, 0);
        else
          tile_mma(acc, s_a(L - 1), 0, kMlpWidth, s_w(L), 0, kMlpWidth, kMlpWidth, 8, 0);
        tc_commit(mbar);
      }
      if (!wait()) break;
      unsigned char *out = sm.a[TRAIN ? (L < 3 ? L : 0) : grp];
#pragma unroll
      for (int c = 0; c < CPT / 16; ++c) {
        const int n0 = c0 + 16 * c;
        float v[16], d[16];
        tmem_ld16(acc + lane_base + n0, v);
        const float4 *bi = reinterpret_cast<const float4 *>(sm.bias[L] + n0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 b = bi[q];
          v[4 * q] += b.x, v[4 * q + 1] += b.y, v[4 * q + 2] += b.z, v[4 * q + 3] += b.w;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          v[i] = gelu<TRAIN>(v[i], &d[i]);
          if (!valid) v[i] = 0.f;
        }
        uint32_t p[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) p[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
        if (L < 3) {
          if (TRAIN) tmem_st16(acc + lane_base + n0, d);
          uint4 *o = reinterpret_cast<uint4 *>(out + tile_offset(row, n0 / 8));
          o[0] = make_uint4(p[0], p[1], p[2], p[3]);
          o[8] = make_uint4(p[4], p[5], p[6], p[7]);
        } else {  // output layer on the rounded activations
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float2 u = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&p[2 * q]));
            const float2 w = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&p[2 * q + 1]));
            const float4 w5 = *reinterpret_cast<const float4 *>(sm.w5 + n0 + 4 * q);
            yp[4 * c + q] = u.x * w5.x + u.y * w5.y + w.x * w5.z + w.y * w5.w;
            if (TRAIN) {
              a4[(8 * c + 2 * q) % (TRAIN ? 16 : 1)] = p[2 * q];
              a4[(8 * c + 2 * q + 1) % (TRAIN ? 16 : 1)] = p[2 * q + 1];
            }
          }
          if (TRAIN)
#pragma unroll
            for (int i = 0; i < 16; ++i) gp[(16 * c + i) % (TRAIN ? 32 : 1)] = d[i];
        }
      }
    }
    if (!ok) break;
    // the 32 sums of a row as a tree over distances 16, 8, 4, 2, 1 (the order in
    // which a warp's butterfly adds them); the halves meet through the shared memory
    // of operands that are done with
    float *sy = reinterpret_cast<float *>(TRAIN ? sm.w[0] : sm.a[grp]);
    float y;
    {
      constexpr int H = TRAIN ? 2 : 1;   // column groups 0 .. H-1 take those H further
      constexpr int M = CPT / 4;
      if (colg >= H)
#pragma unroll
        for (int k = 0; k < M; ++k) sy[((colg - H) * M + k) * kTileM + row] = yp[k];
      group_sync(bar, GT);
      if (colg < H)
#pragma unroll
        for (int k = 0; k < M; ++k) yp[k] += sy[(colg * M + k) * kTileM + row];
      if (TRAIN) {  // distance 8: column groups 0 and 1
        if (colg == 1)
#pragma unroll
          for (int k = 0; k < M; ++k) sy[(2 * M + k) * kTileM + row] = yp[k];
        group_sync(bar, GT);
        if (colg == 0)
#pragma unroll
          for (int k = 0; k < M; ++k) yp[k] += sy[(2 * M + k) * kTileM + row];
      }
#pragma unroll
      for (int o = TRAIN ? 4 : 8; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; ++k) yp[k] += yp[k + o];
      y = yp[0] + b5;
      if (TRAIN) {
        if (colg == 0) sy[3 * M * kTileM + row] = y;
        group_sync(bar, GT);
        y = sy[3 * M * kTileM + row];
      }
    }
    if (!TRAIN) {
      if (colg == 0 && valid) g.y[r0 + row] = y;
      continue;
    }
    if constexpr (TRAIN) {
      // ---- backward
      const float e = valid ? y - t : 0.f;
      const float dy = e * g.inv_n;
      float *a4f = reinterpret_cast<float *>(sm.w[0]);
      float *ph = g.part_h + 2 * blockIdx.x * kMlpPartHead;  // rows of the tile's halves
      if (colg == 0) sm.dy[row] = dy, sm.e[row] = e;
      group_sync(bar, GT);  // and the row sums' scratch is free
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4 *>(sm.w[0] + tile_offset(row, c0 / 8 + c)) =
            make_uint4(a4[4 * c], a4[4 * c + 1], a4[4 * c + 2], a4[4 * c + 3]);
      group_sync(bar, GT);
      // output layer: sums over 64 rows one after the other, a thread per column
      if (tid < 256) {
        const int j = tid & 127, h = tid >> 7;
        const unsigned char *col = sm.w[0] + tile_offset(64 * h, j >> 3) + 2 * (j & 7);
        float s = 0.f;
#pragma unroll 16
        for (int r = 0; r < 64; ++r)
          s = fmaf(sm.dy[64 * h + r],
                   __bfloat162float(*reinterpret_cast<const __nv_bfloat16 *>(col + tile_offset(r, 0))), s);
        ph[h * kMlpPartHead + kMlpWidth + j] = s;
      } else if (tid < 320 && lane < 2) {  // db5 (warp 8), squared errors (warp 9)
        float s = 0.f;
#pragma unroll 16
        for (int r = 0; r < 64; ++r) {
          const int q = 64 * lane + r;
          s = warp == 8 ? s + sm.dy[q] : fmaf(sm.e[q], sm.e[q], s);
        }
        ph[lane * kMlpPartHead + 2 * kMlpWidth + warp - 8] = s;
      }
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = dy * sm.w5[c0 + i] * gp[i];
      group_sync(bar, GT);
      // db4 in the same order, 64 columns at a time through the tile's memory
      // (16-byte pieces of a row at their place XOR the row: no bank conflicts)
#pragma unroll 1
      for (int p = 0; p < 2; ++p) {
        if (colg >> 1 == p)
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<float4 *>(a4f + row * 64 + 4 * ((8 * (colg & 1) + c) ^ (row & 7))) =
                make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
        group_sync(bar, GT);
        if (tid < 128) {
          const int j = tid & 63, h = tid >> 6;
          float s = 0.f;
#pragma unroll 16
          for (int r = 0; r < 64; ++r)
            s += a4f[(64 * h + r) * 64 + 4 * ((j >> 2) ^ (r & 7)) + (j & 3)];
          ph[h * kMlpPartHead + 64 * p + j] = s;
        }
        group_sync(bar, GT);
      }
      // dz of 32 columns to its operand tile; column sums for the bias gradient
      const auto put_dz = [&](unsigned char *dst) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4 *>(dst + tile_offset(row, c0 / 8 + c)) =
              make_uint4(pack_bf16(v[8 * c], v[8 * c + 1]), pack_bf16(v[8 * c + 2], v[8 * c + 3]),
                         pack_bf16(v[8 * c + 4], v[8 * c + 5]), pack_bf16(v[8 * c + 6], v[8 * c + 7]));
      };
      put_dz(sm.w[0]);
      // Weight gradients of the pair's 256 rows are one chain of MMAs: the first
      // CTA's accumulator goes through memory into the second's. In parts (but W1's)
      // four columns of all rows lie together, so that a warp's rows are one run.
      float *pw = g.part_w + (long long)(blockIdx.x / 2) * kMlpPartW;
      const auto chain_in = [&](uint32_t acc, int L) {
        const float *src = pw + (L == 0 ? row * kMlpInPad : mlp_part_w(L) + c0 * kTileM + 4 * row);
        if (L == 0 && colg > 0) return;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (L == 0 && c > 0) break;
          float w[16];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 u = __ldcg(reinterpret_cast<const float4 *>(
                src + (L == 0 ? 4 * q : (16 * c + 4 * q) * kTileM)));
            w[4 * q] = u.x, w[4 * q + 1] = u.y, w[4 * q + 2] = u.z, w[4 * q + 3] = u.w;
          }
          tmem_st16(acc + lane_base + (L == 0 ? 0 : c0 + 16 * c), w);
        }
      };
      const auto chain_out = [&](uint32_t acc, int L) {
        float *dst = pw + (L == 0 ? row * kMlpInPad : mlp_part_w(L) + c0 * kTileM + 4 * row);
        if (L == 0 && colg > 0) return;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (L == 0 && c > 0) break;
          float w[16];
          tmem_ld16(acc + lane_base + (L == 0 ? 0 : c0 + 16 * c), w);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            *reinterpret_cast<float4 *>(dst + (L == 0 ? 4 * q : (16 * c + 4 * q) * kTileM)) =
                make_float4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
        }
      };
      const auto chain_wait = [&](int k) {  // second CTA: the first's k-th output is there
        const bool there = mbar_wait_bounded(&sm.chain[k], 0, g.err, g.wait_limit_ns);
        ok = group_and(bar, GT, there);
        __threadfence();
        return ok;
      };
      const auto chain_signal = [&](int k) {
        if (rank == 1) return;
        group_sync(bar, GT);
        if (tid == 0) {
          __threadfence();
          mbar_arrive_cluster(&sm.chain[k], 1);
        }
      };
      const auto put_columns = [&](int L) {  // the four quadrants' column sums
        if (tid < kMlpWidth)
          g.part_b[(long long)blockIdx.x * 3 * kMlpWidth + L * kMlpWidth + tid] =
              ((sm.colsum[0][tid] + sm.colsum[1][tid]) + sm.colsum[2][tid]) + sm.colsum[3][tid];
      };
      // dz_L = da_L gelu'(z_L), da_L in acc_d
      const uint32_t acc_d = tmem + 384u;
      const auto next_dz = [&](int L, unsigned char *dst) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float d[16], q[16];
          tmem_ld16(acc_d + lane_base + c0 + 16 * c, d);
          tmem_ld16(tmem + 128u * L + lane_base + c0 + 16 * c, q);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[16 * c + i] = valid ? d[i] * q[i] : 0.f;
        }
        put_dz(dst);
        sm.colsum[quad][c0 + lane] = column_sums(v);
      };
      // Layers 0..3; dz takes the memory of what it makes needless: dz3 is in W1's,
      // dz2 goes to W3's, dz1 to a2's, dz0 to a1's, and W1 comes back in dz3's. The
      // accumulators of the weight gradients take those of the gelu' just used.
      ready();
      if (gt == 0) {
        tile_mma(acc_d, s_w(1), 0, kMlpWidth, s_w(3), 1, kMlpWidth, kMlpWidth, 8, 0);
        tc_commit(mbar);
      }
      if (!wait()) break;
      next_dz(2, sm.w[2]);
#pragma unroll 1
      for (int k = 0; k < 3; ++k) {  // dW3 and da1, dW2 and da0, dW1 and dW0
        const uint32_t acc_w = tmem + 128u * (2 - k);
        const uint32_t dz_old = k == 0 ? s_w(1) : k == 1 ? s_w(3) : s_a(2);
        const uint32_t dz = k == 0 ? s_w(3) : k == 1 ? s_a(2) : s_a(1);
        if (rank == 1) {
          if (!chain_wait(k)) break;
          chain_in(acc_w, 3 - k);
          if (k == 2) chain_in(acc_d, 0);
        }
        if (k == 1) cp_async_wait_all();
        ready();
        if (gt == 0) {
          tile_mma(acc_w, dz_old, 1, kMlpWidth, s_a(2 - k), 1, kMlpWidth, kMlpWidth, 8, rank);
          if (k < 2)
            tile_mma(acc_d, dz, 0, kMlpWidth, k == 0 ? s_w(2) : s_w(1), 1, kMlpWidth, kMlpWidth, 8, 0);
          else
            tile_mma(acc_d, dz, 1, kMlpWidth, s_x, 1, kMlpInPad, kMlpInPad, 8, rank);
          tc_commit(mbar);
        }
        put_columns(2 - k);
        if (!wait()) break;
        if (k == 0) load_weights<kMlpWidth>(sm.w[0], g.wbf + mlp_off_w(1));
        chain_out(acc_w, 3 - k);
        if (k == 2) chain_out(acc_d, 0);
        chain_signal(k);
        if (k < 2) next_dz(1 - k, sm.a[2 - k]);
      }
    }
    if (TRAIN) break;
  }
  // a wait ran out: one more bounded wait for the MMAs in flight
  if (!ok && gt == 0) mbar_wait_bounded(mbar, phase ^ 1u, g.err, g.wait_limit_ns);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(sm.tmem_slot, kCols);
  // the first CTA's last signal has reached the second's shared memory
  if constexpr (TRAIN) cooperative_groups::this_cluster().sync();
}

// Sums the gradients' parts in order; Adam (with bias corrections c1 = 1 - b1^t,
// c2 = 1 - b2^t and decoupled weight decay wd) or the gradient itself. The last
// element is the loss.
__global__ void mlp_update(const MlpUpdateArgs a) {
  after_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > kMlpLoss) return;
  const float *p;
  long long stride;
  int count;
  if (i >= mlp_off_b(3)) {  // b4, w5, b5, loss: parts of 64 rows
    p = a.part_h + (i - mlp_off_b(3)), stride = kMlpPartHead, count = 2 * a.tiles;
  } else {
    const int L = i < mlp_off_w(1) ? 0 : 1 + (i - mlp_off_w(1)) / 16512;
    if (i >= mlp_off_b(L))  // of a tile
      p = a.part_b + L * kMlpWidth + (i - mlp_off_b(L)), stride = 3 * kMlpWidth, count = a.tiles;
    else {  // of a pair of tiles, four columns of all rows together (but for W1)
      const int t = i - mlp_off_w(L);
      p = a.part_w + mlp_part_w(L) + t, stride = kMlpPartW, count = (a.tiles + 1) / 2;
      if (L > 0) i = mlp_off_w(L) + ((t >> 2) & 127) * kMlpWidth + (t >> 9) * 4 + (t & 3);
    }
  }
  float s = 0.f;
#pragma unroll 8
  for (int k = 0; k < count; ++k) s += p[k * stride];
  if (i == kMlpLoss) {
    *a.loss = s * a.loss_scale;
    return;
  }
  if (a.grad) {
    a.grad[i] = s;
    return;
  }
  const float mi = fmaf(a.b1, a.m[i], (1.f - a.b1) * s);
  const float vi = fmaf(a.b2, a.v[i], (1.f - a.b2) * s * s);
  a.m[i] = mi;
  a.v[i] = vi;
  float th = a.theta[i];
  th -= a.lr * ((mi / a.c1) / (sqrtf(vi / a.c2) + a.eps) + a.wd * th);
  a.theta[i] = th;
  a.theta_bf[i] = __float2bfloat16_rn(th);
}

__global__ void mlp_to_bf16(const float *__restrict__ theta, __nv_bfloat16 *__restrict__ theta_bf,
                            long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) theta_bf[i] = __float2bfloat16_rn(theta[i]);
}

unsigned blocks(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

template <bool TRAIN>
cudaError_t launch_net(const MlpNetArgs &g, int grid, cudaStream_t s) {
  const int smem = (int)sizeof(NetSmem<TRAIN>);
  const cudaError_t e =
      cudaFuncSetAttribute(mlp_net<TRAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3(kNetThreads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 2;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  c.attrs = at;
  c.numAttrs = TRAIN ? 2 : 1;
  return cudaLaunchKernelEx(&c, mlp_net<TRAIN>, g);
}

}  // namespace

int mlp_tiles(long long n) { return (int)((n + kTileM - 1) / kTileM); }

cudaError_t launch_mlp_forward(const MlpNetArgs &g, int sms, cudaStream_t s) {
  if (g.n <= 0) return cudaSuccess;
  const int tiles = mlp_tiles(g.n);
  return launch_net<false>(g, tiles < sms ? tiles : sms, s);
}

cudaError_t launch_mlp_gradient(const MlpNetArgs &g, cudaStream_t s) {
  if (g.n <= 0) return cudaErrorInvalidValue;
  return launch_net<true>(g, (mlp_tiles(g.n) + 1) / 2 * 2, s);
}

cudaError_t launch_mlp_update(const MlpUpdateArgs &a, cudaStream_t s) {
  return launch_after(mlp_update, blocks(kMlpLoss + 1, 128), 128, 0, s, a);
}

cudaError_t launch_mlp_to_bf16(const float *theta, __nv_bfloat16 *theta_bf, long long n,
                               cudaStream_t s) {
  mlp_to_bf16<<<blocks(n, 256), 256, 0, s>>>(theta, theta_bf, n);
  return cudaGetLastError();
}

}  // namespace winds
