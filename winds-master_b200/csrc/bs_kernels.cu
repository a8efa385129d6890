// bs_kernels.cu -- sm_100a kernels of the induced-velocity (Biot-Savart) direct
// sum that replaces core/BiotSavart.m:80-116 and the BiotSavart_naive /
// BiotSavart_sh kernels of cuda/source/BiotSavartMex.cu:131-193.
//
// Kernels
//   bs_begin           counters and bounding box at the start of an evaluation
//   bs_chain_count,    MATLAB-layout F1/F2/gamma/rc -> 64-byte records (+ FP64
//   bs_pack            copies), the device-side replacement of the host crunch_f
//                      / crunch_rg packing (BiotSavartMex.cu:316-357), in input
//                      order or laid out along the wake's lines of filaments
//                      (x2 of a record = x1 of the one before, but for marked
//                      heads where a line starts or the input has no link)
//                      and MATLAB-layout P -> double4 targets (crunch_p, :361-379)
//   bs_f32c            persistent FP32 direct sum on independent warp workers:
//                      each warp stages its filament tiles into its own shared
//                      memory by bulk copies (cp.async.bulk + mbarrier), keeps
//                      T register-resident targets per lane, Kahan-compensates
//                      the per-target sums, and recomputes the near-singular
//                      pairs in FP64 with all 32 lanes; each interaction
//                      reuses the previous record's endpoint rsqrt, and groups
//                      distant from the warp's targets run in an expanded form
//   bs_target_keys     places on a Hilbert curve (the order: bs_sort.cuh)
//   bs_f64             FP64 direct sum: short forms of the terms, or the reference's
//                      sequence in order
//   bs_reduce          deterministic sum of the per-chunk partials, written in
//                      MATLAB layout (reassem_uind, :383-401)
//   bs_length          filament lengths (core/FilamentLength.m:27-44)
#include "bs_device.cuh"
#include "bs_launch.h"
#include "bs_sort.cuh"
#include "bs_types.h"

#include <cfloat>
#include <type_traits>

#include <cub/device/device_radix_sort.cuh>

namespace winds {

// --------------------------------------------------------------- packing
__global__ void bs_begin(BBox *bb, unsigned *ctr, unsigned long long *near,
                         unsigned long long *cnt) {
  after_previous();
  begin_evaluation(bb, ctr);
  if (threadIdx.x < 2) near[threadIdx.x] = 0ull;
  if (threadIdx.x < 2 * kPackFams) cnt[threadIdx.x] = 0ull;
}

// WInDS's filaments meet at the wake's nodes: the shed call's F2(i) is its
// F1(i+1) (WInDS.m:150, along the first index) and the trailing call's
// F2(:,:,j) is its F1(:,:,j-1) (WInDS.m:153, along the third). The FP32 records
// go along such a line, each with the end it shares with its predecessor as its
// second end, so that the kernel reuses the predecessor's endpoint term
// (interact). Two orders: the input's own (a chain along the first index), and,
// where the family has more links along the third index, line by line along
// that one. bs_chain_count counts, per family, the filaments whose end is
// bitwise the start of their neighbour along each index. A record whose end is
// not its predecessor's is a head (marked in the record): the kernel evaluates
// the end from its own L, so any input is evaluated correctly.
__device__ __forceinline__ bool same_point(const double *__restrict__ F2, long long b2,
                                           const double *__restrict__ F1, long long b1,
                                           long long d0) {
  return F2[b2] == F1[b1] && F2[b2 + d0] == F1[b1 + d0] && F2[b2 + 2 * d0] == F1[b1 + 2 * d0];
}

// Up to kPackFams families per launch, each with its run of blocks.
__global__ void bs_chain_count(const PackArgs a) {
  after_previous();
  int k = 0;
  while (k + 1 < a.nfam && (int)blockIdx.x >= a.fam[k + 1].block0) ++k;
  const PackArgs::Fam &m = a.fam[k];
  const long long f = (long long)(blockIdx.x - m.block0) * blockDim.x + threadIdx.x;
  bool s = false, t = false;
  if (f < m.nf) {
    const long long d0 = m.d0, jb = f / d0, i = f - jb * d0, j = jb % m.d2;
    const long long b = i + d0 * 3 * jb;
    if (i + 1 < d0) s = same_point(m.F2, b, m.F1, b + 1, d0);   // F2(i) == F1(i+1)
    if (j >= 1) t = same_point(m.F2, b, m.F1, b - 3 * d0, d0);  // F2(:,:,j) == F1(:,:,j-1)
  }
  const unsigned ns = __popc(__ballot_sync(0xffffffffu, s));
  const unsigned nt = __popc(__ballot_sync(0xffffffffu, t));
  if ((threadIdx.x & 31) == 0) {
    if (ns) atomicAdd(m.cnt, (unsigned long long)ns);
    if (nt) atomicAdd(m.cnt + 1, (unsigned long long)nt);
  }
}

// One thread per filament of a family, in input order; its record goes to slot
// off + f, or (cnt given and cnt[1] > cnt[0]) to its place along the third
// index. The blocks past the families fill [pad_from, pad_to) with inert
// filaments (far away, zero length, zero circulation), those past them pack the
// targets of a MATLAB array P [ns, 3, ...].
__global__ void bs_pack(const PackArgs a) {
  after_previous();
  float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  if ((int)blockIdx.x >= a.tgt_block0) {
    const long long t = (long long)(blockIdx.x - a.tgt_block0) * blockDim.x + threadIdx.x;
    if (t < a.nt) {
      const long long j = t / a.ns, b = t - j * a.ns + a.ns * 3 * j;
      const double x = a.P[b], y = a.P[b + a.ns], z = a.P[b + 2 * a.ns];
      a.tp_raw[t] = make_double4(x, y, z, 0.0);
      if (a.tgroup) a.tgroup[t] = 0;
      lo[0] = hi[0] = (float)x, lo[1] = hi[1] = (float)y, lo[2] = hi[2] = (float)z;
    }
    bbox_accumulate(lo, hi, a.bb->tmin, a.bb->tmax);
    return;
  }
  if ((int)blockIdx.x >= a.pad_block0) {
    const long long f =
        a.pad_from + (long long)(blockIdx.x - a.pad_block0) * blockDim.x + threadIdx.x;
    if (f < a.pad_to) pack_inert(f, a.pk, a.ra, a.rb);
    return;
  }
  int k = 0;
  while (k + 1 < a.nfam && (int)blockIdx.x >= a.fam[k + 1].block0) ++k;
  const PackArgs::Fam &m = a.fam[k];
  const long long f = (long long)(blockIdx.x - m.block0) * blockDim.x + threadIdx.x;
  if (f < m.nf) {
    const bool along3 = m.cnt && m.cnt[1] > m.cnt[0];
    const long long d0 = m.d0, jb = f / d0, i = f - jb * d0;
    const long long b = i + d0 * 3 * jb;
    const double x1 = m.F1[b], y1 = m.F1[b + d0], z1 = m.F1[b + 2 * d0];
    const double x2 = m.F2[b], y2 = m.F2[b + d0], z2 = m.F2[b + 2 * d0];
    long long slot = m.off + f;
    bool head;
    if (along3) {
      const long long bl = jb / m.d2, j = jb - bl * m.d2;
      slot = m.off + j + m.d2 * (i + d0 * bl);
      head = !(j >= 1 && same_point(m.F2, b, m.F1, b - 3 * d0, d0));
    } else {
      head = !(i >= 1 && same_point(m.F2, b - 1, m.F1, b, d0));
    }
    pack_filament(slot, x1, y1, z1, x2, y2, z2, m.gam[f], m.rc[f], !along3, head, a.model, a.dcut,
                  a.pk, a.ra, a.rb);
    lo[0] = (float)fmin(x1, x2), lo[1] = (float)fmin(y1, y2), lo[2] = (float)fmin(z1, z2);
    hi[0] = (float)fmax(x1, x2), hi[1] = (float)fmax(y1, y2), hi[2] = (float)fmax(z1, z2);
  }
  bbox_accumulate(lo, hi, a.bb->fmin, a.bb->fmax);
}

// Sort key of a target: group id above the 30-bit Hilbert position in the
// targets' bounding box (bit 30: the target is unused, and sorts after every
// live target of its group); for counting, the position's leading 24 bits, of which
// the last value is the unused targets' (kUnusedKey, bs_sort.cuh).
template <class KEY>
__global__ void bs_target_keys(const double4 *__restrict__ tp, const int *__restrict__ tgroup,
                               long long n, const BBox *bb, KEY *keys, int *vals) {
  after_previous();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const double4 p = tp[t];
  const double q[3] = {p.x, p.y, p.z};
  const float lo[3] = {key_float(bb->tmin[0]), key_float(bb->tmin[1]), key_float(bb->tmin[2])};
  const float hi[3] = {key_float(bb->tmax[0]), key_float(bb->tmax[1]), key_float(bb->tmax[2])};
  const unsigned h = hilbert_key(q, lo, hi);
  if constexpr (sizeof(KEY) == 4 && !std::is_integral<KEY>::value) {
    keys[t] = p.w != 0.0 ? kUnusedKey : fminf((float)(h >> 6), kUnusedKey - 1.f);  // 8 bits a coordinate
  } else {
    KEY code = h;
    if (p.w != 0.0) code |= (KEY)1 << 30;
    if (sizeof(KEY) == 8) code |= (KEY)(unsigned)tgroup[t] << 31;
    keys[t] = code;
    vals[t] = (int)t;
  }
}

__global__ void bs_gather_targets(const double4 *__restrict__ src, const int *__restrict__ perm,
                                  long long n, double4 *dst) {
  after_previous();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) dst[t] = src[perm[t]];
}

// Largest possible squared target-endpoint distance from the bounds; the
// reach cut-off can only zero a term when co^2 is below it.
__device__ __forceinline__ bool co_can_trigger(const BBox *bb, double co) {
  double d2 = 0.0;
  for (int c = 0; c < 3; ++c) {
    const double a = (double)key_float(bb->tmax[c]) - (double)key_float(bb->fmin[c]);
    const double b = (double)key_float(bb->fmax[c]) - (double)key_float(bb->tmin[c]);
    const double m = fmax(fabs(a), fabs(b)) * (1.0 + 1e-6) + 1e-3;
    d2 += m * m;
  }
  return co * co < d2;  // false for NaN co: r > NaN is never true
}

// Cuts a work item to the live part of its group (GroupLive): the tile to its
// live targets, the filament range to the live filaments. False when nothing
// of the item is live; its partial sums are then neither written nor read.
__device__ __forceinline__ bool clip_live(const GroupLive *live, Item &it, Tile &tl) {
  const GroupLive gl = live[tl.group];
  const long long tn = gl.t_end - tl.t_begin;
  if (tn <= 0 || it.f_begin >= gl.f_end) return false;
  if (tn < tl.t_count) tl.t_count = (int)tn;
  if (it.f_end > gl.f_end) it.f_end = gl.f_end;
  return true;
}

// ------------------------------------------------------- FP32 direct sum
// Every warp is an independent worker: it takes work items (a tile of 32 x T
// targets against a filament range) from the persistent queue by itself and
// streams the range through its own ring of shared-memory stages, so warps
// never wait for one another (no CTA barrier in the kernel). A CTA holds kWarps
// workers that share nothing but the SM.
constexpr int kWarps = 4;
constexpr int kThreads = 32 * kWarps;
constexpr uint64_t kDefaultWaitNs = 2000000000ull;  // 2 s per tile: far above any real latency

template <int KF>
struct StageSmem {
  static constexpr int kBytes = KF * 64;
  // two stages: a warp's tile takes ~5-50 us, a bulk copy ~2 us
  static constexpr int kStages = 2;
};

// Shared memory of one worker: its filament stages, the Kahan state of its
// targets (sum, compensation) x 3 components as floats, the targets themselves
// relative to their lane's centre (component c of the lane's target t at
// (c T + t) 32 + lane), the near-singular bits of the current tile (a word per
// lane and group of four filaments), its full[s] barriers (bytes landed) and its target ball
// (centre, radius, threshold).
template <int T>
struct NearBits {
  using type = unsigned;  // bit 8 j + t: filament j of the group, target t
  static constexpr int kPer = 8;
};
template <>
struct NearBits<2> {
  using type = unsigned short;
  static constexpr int kPer = 4;
};
template <>
struct NearBits<4> {
  using type = unsigned short;
  static constexpr int kPer = 4;
};

template <int T, int KF>
__host__ __device__ constexpr size_t warp_smem_bytes() {
  constexpr int S = StageSmem<KF>::kStages;
  return ((size_t)S * StageSmem<KF>::kBytes + (size_t)9 * 32 * T * sizeof(float) +
          (size_t)(KF / 4) * 32 * sizeof(typename NearBits<T>::type) + S * sizeof(uint64_t) + 8 * sizeof(float) +
          127) / 128 * 128;
}

template <int T, int KF>
__host__ __device__ constexpr size_t f32c_smem_bytes_t() {
  return kWarps * warp_smem_bytes<T, KF>();
}

// Kahan step: (sum, comp) += v.
__device__ __forceinline__ void kahan_add(float &sum, float &comp, float v) {
  const float y = __fsub_rn(v, comp);
  const float s = __fadd_rn(sum, y);
  comp = __fsub_rn(__fsub_rn(s, sum), y);
  sum = s;
}

// Hands filaments f0 .. f0+KF to the copy engine into `stage`, completing on `bar`.
template <int KF>
__device__ __forceinline__ void issue_stage(const F32cArgs &a, unsigned char *stage, uint64_t *bar,
                                            int f0) {
  mbar_arrive_expect_tx(bar, StageSmem<KF>::kBytes);
  bulk_g2s(stage, a.pk + (size_t)f0 * 4, KF * 64, bar);
}

// Orders this thread's earlier shared-memory accesses (generic proxy) before
// later bulk copies into the same bytes (async proxy).
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ----------------------------------------------------- packed FP32 arithmetic
// The direct sum runs on pairs of targets: every FP32 operation is a packed
// f32x2 instruction (two independent IEEE operations, round to nearest) on two
// of a lane's targets, so one issue slot does two interactions' worth of
// arithmetic. A filament's field goes to both halves of the instruction from
// one register (bc costs no instruction), and a target holds 12 registers: with
// the filaments in the two halves instead, the broadcast targets and the
// double sums took 24 a target and capped the kernel at three warps a
// scheduler, where latency, not the FMA pipe, bounded it.
__device__ __forceinline__ float2 bc(const float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 neg2(const float2 v) { return make_float2(-v.x, -v.y); }
__device__ __forceinline__ float2 rsqrt2(const float2 v) {
  return make_float2(rsqrt_approx(v.x), rsqrt_approx(v.y));
}
__device__ __forceinline__ float2 rcp2(const float2 v) {
  return make_float2(rcp_approx(v.x), rcp_approx(v.y));
}

// One filament of a stage, relative to this lane's centre c.
struct Fil {
  float qx, qy, qz;  // x1 - c (from the hi/lo split)
  float Lx, Ly, Lz, L2, D;
  float Mx, My, Mz;  // K L, K = gamma/4pi
  float Rn2;         // near-singular threshold (careful path)
};

// Filament record (4 float4, layout in bs_types.h) whose chunk q is at r[q ^ sw].
__device__ __forceinline__ Fil load_filament(const float4 *r, int sw, float cx, float cy,
                                             float cz) {
  const float4 a = r[0 ^ sw], b = r[1 ^ sw], c = r[2 ^ sw], d = r[3 ^ sw];
  Fil f;
  f.qx = (a.x - cx) + c.x;
  f.qy = (a.y - cy) + c.y;
  f.qz = (a.z - cz) + c.z;
  f.L2 = fabsf(a.w);
  f.Mx = b.x, f.My = b.y, f.Mz = b.z;
  f.Rn2 = c.w;
  f.Lx = d.x, f.Ly = d.y, f.Lz = d.z, f.D = d.w;
  return f;
}

// Two targets against one filament, added to (ax, ay, az) (one half per
// target). (npx, npy, npz) = -(P - c). With near_some, terms with r1.r2 < Rn2 are
// zeroed and recorded in `bits` (bit0 for the pair's first target, bit1 for its
// second); they are redone in FP64 after the tile. With co_on the terms beyond
// the reach cut-off (both ends farther than co2, squared) are zeroed for good.
//
// The filaments form chains: x2 of a record is x1 of the record before it --
// the wake's filaments meet at its nodes -- so 1/|x2 - P| is the previous
// record's 1/|x1 - P|, carried in `ti`, and a record needs no rsqrt for it.
// Before a record that starts a chain, chain_start puts 1/|x2 - P| into the
// carry. 1/|x1 - P| is left there for the next record.
template <int MODEL>
__device__ __forceinline__ void interact(float2 npx, float2 npy, float2 npz, const Fil &f,
                                         float Rn2, bool near_some, float co2, bool co_on,
                                         float2 &ax, float2 &ay, float2 &az, unsigned &bits,
                                         unsigned bit0, unsigned bit1, float2 &ti) {
  const float2 nx = __fadd2_rn(bc(f.qx), npx);  // x1 - P = -r1
  const float2 ny = __fadd2_rn(bc(f.qy), npy);
  const float2 nz = __fadd2_rn(bc(f.qz), npz);
  float2 r1s = __fmul2_rn(nx, nx);
  r1s = __ffma2_rn(ny, ny, r1s);
  r1s = __ffma2_rn(nz, nz, r1s);
  float2 ld = __fmul2_rn(bc(f.Lx), nx);  // -L.r1
  ld = __ffma2_rn(bc(f.Ly), ny, ld);
  ld = __ffma2_rn(bc(f.Lz), nz, ld);
  const float2 dot = __fadd2_rn(r1s, ld);  // r1 . r2
  const float2 i1 = rsqrt2(r1s), i2 = ti;
  const float2 gg = __fmul2_rn(i1, i2);
  const float2 e = __ffma2_rn(dot, gg, bc(1.f));  // 1 + cos(theta)
  // K (r1 x r2) = K L x r1 = (x1 - P) x (K L): no cancellation for far or
  // collinear points
  const float2 cx = __ffma2_rn(ny, bc(f.Mz), __fmul2_rn(nz, bc(-f.My)));
  const float2 cy = __ffma2_rn(nz, bc(f.Mx), __fmul2_rn(nx, bc(-f.Mz)));
  const float2 cz = __ffma2_rn(nx, bc(f.My), __fmul2_rn(ny, bc(-f.Mx)));
  float2 ub;
  if (MODEL == kCoreVatistas) {
    // Cnu / (r1 r2 (r1 r2 + r1.r2)) with h^2 = |L x r1|^2/|L|^2 and rc^4 folded:
    // Cnu = |c|^2 / sqrt(|c|^4 + D), c = K L x r1, D = (K^2 rc^2 |L|^2)^2
    float2 c2 = __fmul2_rn(cx, cx);
    c2 = __ffma2_rn(cy, cy, c2);
    c2 = __ffma2_rn(cz, cz, c2);
    const float2 q = __ffma2_rn(c2, c2, bc(f.D));
    const float2 w = __fmul2_rn(__fmul2_rn(__fadd2_rn(i1, i2), gg), c2);
    ub = __fmul2_rn(w, rsqrt2(__fmul2_rn(__fmul2_rn(e, e), q)));
  } else {
    // (r1+r2)/(r1r2(r1r2+r1.r2) + d|L|^2) = (i1+i2) gg / (e + d|L|^2 gg^2)
    ub = __fmul2_rn(__fmul2_rn(__fadd2_rn(i1, i2), gg),
                    rcp2(__ffma2_rn(bc(f.D), __fmul2_rn(gg, gg), e)));
  }
  if (co_on) {  // uniform over the launch
    const float2 r2s = __fadd2_rn(dot, __fadd2_rn(bc(f.L2), ld));  // |r1 - L|^2
    if (fminf(r1s.x, r2s.x) > co2) ub.x = 0.f;
    if (fminf(r1s.y, r2s.y) > co2) ub.y = 0.f;
  }
  if (near_some) {  // uniform over the warp
    if (dot.x < Rn2) {
      bits |= bit0;
      ub.x = 0.f;
    }
    if (dot.y < Rn2) {
      bits |= bit1;
      ub.y = 0.f;
    }
  }
  ax = __ffma2_rn(ub, cx, ax);
  ay = __ffma2_rn(ub, cy, ay);
  az = __ffma2_rn(ub, cz, az);
  ti = i1;
}

// The carry of a record that starts a chain: 1/|x2 - P| from its own x1 and L.
template <int NP>
__device__ __forceinline__ void chain_start(const Fil &f, const float2 (&npx)[NP],
                                            const float2 (&npy)[NP], const float2 (&npz)[NP],
                                            float2 (&ti)[NP]) {
  const float ex = f.qx + f.Lx, ey = f.qy + f.Ly, ez = f.qz + f.Lz;
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const float2 nx = __fadd2_rn(bc(ex), npx[p]), ny = __fadd2_rn(bc(ey), npy[p]),
                 nz = __fadd2_rn(bc(ez), npz[p]);
    float2 r2s = __fmul2_rn(nx, nx);
    r2s = __ffma2_rn(ny, ny, r2s);
    r2s = __ffma2_rn(nz, nz, r2s);
    ti[p] = rsqrt2(r2s);
  }
}

// ------------------------------------------------------------ distant form
// A filament is distant when its endpoints are at least kDistantRatio radii
// from the centre w of the ball of the warp's targets (and it is far, as the
// screen defines it). Everything is then expanded about w. With q = x1 - w,
// p = P - w, r1 = |x1 - P|, r2 = |x2 - P|, M = K L:
//     |x1 - P|^2  = |q|^2 + |p|^2 - 2 q.p                       (4 operations)
//     r1r2 + r1.r2 = ((r1 + r2)^2 - |L|^2) / 2                  (no dot product)
//     K L x r1     = q x M - p x M
// |q|^2, q x M and the rest are per filament and warp, not per lane: each lane
// prepares one filament of the 32 it screens, in place of the record's fields
// that the loop no longer needs.
//
// Core-free filaments, whose core changes no term by more than the roundoff
// that forming the term has anyway, go further: the sum over filaments of
// ub (x1 - P) x M is  B - p x A  with A = sum ub M, B = sum ub (q x M), so the
// cross product leaves the pair loop, and an interaction costs 16 FP32
// operations and two MUFU results, against 33 and 6 per filament and lane in
// the form above. With the core it costs 28 (Vatistas, whose factor needs
// |K L x r1|^2) or 17 (cut-off).
//   Vatistas  the factor 1/sqrt(1 + (rc/h)^4), h the distance from the
//             filament's line, is short of 1 by at most (rc/h)^4 / 2 and the
//             term's cross product is |M| h, so leaving it out moves the term
//             by ub |M| rc^4 / (2 h^3), where rounding moves it by about
//             2^-24 ub |M| r: kCoreFree4 rc^4 <= h^3 max(h, r) (54^4 is 2^23).
//   cut-off   every target is at least r from it with r^4 >= 2^24 d |L|^2, so
//             the denominator's d |L|^2 gg^2 <= 2^-24 <= 2^-24 e (e >= 1 there).
// Rounding: |x1 - P|^2 is formed from terms of at most |q|^2 + 2|q||p| + |p|^2
// with |p| <= |q| / kDistantRatio. The form is the more exact one: with it at three
// radii the error against FP64 (2-norm, wakes of 3k to 175k filaments, steps of one to
// eight rotors) is 2 to 15% larger, and the core left out or not makes no difference.
constexpr float kDistantRatio = 1.5f;
// squared distances for which no product of the form leaves FP32's range, and
// |M|^2 |q|^2 for which the fourth power of the cross product does not
constexpr float kDistantMinSq = 1e-12f, kDistantMaxSq = 1e16f, kDistantMaxMq = 1e17f;
constexpr float kCoreFree4 = 54.f * 54.f * 54.f * 54.f;
constexpr float kCutoffFreeSq = 4096.f;  // r^2 >= 4096 sqrt(d |L|^2) is r^4 >= 2^24 d |L|^2

// One prepared filament against the lane's 2 NP targets: (mx, my, mz) = -2 p,
// p2 = |p|^2. a = q, |q|^2; c = 2 q x M; b = 2 M, -|L|^2, but for the Vatistas
// core M, -|L|^2; D = 16 (K^2 rc^2 |L|^2)^2 or 2 d |L|^2. (Ax, Ay, Az) = A, B is
// added to (ax, ay, az). Carry: 1/r1, r1. CORE: kNoCore or the kernel's model.
constexpr int kNoCore = 2;
template <int NP, int CORE>
__device__ __forceinline__ void distant_filament(const float4 a, const float4 b, const float4 c,
                                                 const float D, const float2 (&mx)[NP],
                                                 const float2 (&my)[NP], const float2 (&mz)[NP],
                                                 const float2 (&p2)[NP], float2 (&ax)[NP],
                                                 float2 (&ay)[NP], float2 (&az)[NP],
                                                 float2 (&Ax)[NP], float2 (&Ay)[NP],
                                                 float2 (&Az)[NP], float2 (&ti)[NP],
                                                 float2 (&tr)[NP]) {
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    float2 r1s = __fadd2_rn(bc(a.w), p2[p]);
    r1s = __ffma2_rn(bc(a.x), mx[p], r1s);
    r1s = __ffma2_rn(bc(a.y), my[p], r1s);
    r1s = __ffma2_rn(bc(a.z), mz[p], r1s);
    const float2 i1 = rsqrt2(r1s);
    const float2 r1 = __fmul2_rn(r1s, i1);
    const float2 s = __fadd2_rn(r1, tr[p]);
    const float2 y = __ffma2_rn(s, s, bc(b.w));  // 2 (r1r2 + r1.r2)
    const float2 gg = __fmul2_rn(i1, ti[p]);
    ti[p] = i1;
    tr[p] = r1;
    if (CORE == kCoreVatistas) {
      // 2 K L x r1 and its squared length; s gg^2 / (y gg) |c|^2 / sqrt(|c|^4 + D)
      const float2 cx = __ffma2_rn(my[p], bc(b.z), __ffma2_rn(mz[p], bc(-b.y), bc(c.x)));
      const float2 cy = __ffma2_rn(mz[p], bc(b.x), __ffma2_rn(mx[p], bc(-b.z), bc(c.y)));
      const float2 cz = __ffma2_rn(mx[p], bc(b.y), __ffma2_rn(my[p], bc(-b.x), bc(c.z)));
      float2 c2 = __fmul2_rn(cx, cx);
      c2 = __ffma2_rn(cy, cy, c2);
      c2 = __ffma2_rn(cz, cz, c2);
      const float2 q = __ffma2_rn(c2, c2, bc(D));
      const float2 yg = __fmul2_rn(y, gg);
      const float2 ub = __fmul2_rn(__fmul2_rn(__fmul2_rn(s, gg), __fmul2_rn(gg, c2)),
                                   rsqrt2(__fmul2_rn(__fmul2_rn(yg, yg), q)));
      ax[p] = __ffma2_rn(ub, cx, ax[p]);
      ay[p] = __ffma2_rn(ub, cy, ay[p]);
      az[p] = __ffma2_rn(ub, cz, az[p]);
    } else {
      const float2 den = CORE == kCoreCutoff ? __ffma2_rn(bc(D), gg, y) : y;
      const float2 ub = __fmul2_rn(__fmul2_rn(s, gg), rcp2(den));
      Ax[p] = __ffma2_rn(ub, bc(b.x), Ax[p]);
      Ay[p] = __ffma2_rn(ub, bc(b.y), Ay[p]);
      Az[p] = __ffma2_rn(ub, bc(b.z), Az[p]);
      ax[p] = __ffma2_rn(ub, bc(c.x), ax[p]);
      ay[p] = __ffma2_rn(ub, bc(c.y), ay[p]);
      az[p] = __ffma2_rn(ub, bc(c.z), az[p]);
    }
  }
}

// The carry of a prepared filament that starts a chain: 1/r2 and r2 of its own
// second endpoint q + L.
template <int NP>
__device__ __forceinline__ void distant_start(const float4 a, const float4 d,
                                              const float2 (&mx)[NP], const float2 (&my)[NP],
                                              const float2 (&mz)[NP], const float2 (&p2)[NP],
                                              float2 (&ti)[NP], float2 (&tr)[NP]) {
  const float ex = a.x + d.x, ey = a.y + d.y, ez = a.z + d.z;
  const float e2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    float2 r2s = __fadd2_rn(bc(e2), p2[p]);
    r2s = __ffma2_rn(bc(ex), mx[p], r2s);
    r2s = __ffma2_rn(bc(ey), my[p], r2s);
    r2s = __ffma2_rn(bc(ez), mz[p], r2s);
    ti[p] = rsqrt2(r2s);
    tr[p] = __fmul2_rn(r2s, ti[p]);
  }
}

// Bits 0, 4, ..., 28 of x gathered into bits 0 .. 7.
__device__ __forceinline__ unsigned gather_nibbles(unsigned x) {
  x = (x | (x >> 3)) & 0x03030303u;
  x = (x | (x >> 6)) & 0x000f000fu;
  return (x | (x >> 12)) & 0xffu;
}
__device__ __forceinline__ unsigned nibble_any(unsigned m) {
  m |= m >> 2;
  return gather_nibbles((m | (m >> 1)) & 0x11111111u);
}
__device__ __forceinline__ unsigned nibble_all(unsigned m) { return nibble_any(~m) ^ 0xffu; }

// A near-singular pair of a tile, listed in the tile's consumed stage: the
// FP64 reference term `u` of filament `fidx` at the owner's target `slot`.
struct NearEntry {
  double u[3];
  int fidx, slot;
};

// One item: the lane's T targets (T even) against filaments [it.f_begin,
// it.f_end), streamed through the warp's S stages (tile g of the warp in stage
// g % S). Returns false, for the whole warp, when a bounded wait ran out (the
// item is abandoned after the copies in flight have landed).
template <int T, int KF, int MODEL>
__device__ __forceinline__ bool f32c_item(const F32cArgs &a, const Item &it, unsigned char *stages,
                                          uint64_t *full, float *s_k, const float *s_p,
                                          typename NearBits<T>::type *s_nb, unsigned &gt, float cx, float cy,
                                          float cz, float S2, const float *ws, bool co_on,
                                          unsigned &near_cnt, unsigned long long &free_cnt,
                                          const Tile &tl) {
  constexpr int S = StageSmem<KF>::kStages;
  constexpr int kB = StageSmem<KF>::kBytes;
  constexpr int NP = T / 2;
  constexpr int kPer = NearBits<T>::kPer;
  constexpr unsigned kGroups = (1u << (KF / 4)) - 1u;
  const int lane = threadIdx.x & 31;
  const int ntiles = (it.f_end - it.f_begin) / KF;
  const float co2 = (float)(a.co * a.co);
  const int nslots = tl.t_count - lane * T;  // this lane's targets in the tile
  const unsigned live_slots = (unsigned)(nslots < 0 ? 0 : (nslots > T ? T : nslots));
  RefParams rp;
  rp.model = a.model;
  rp.d = a.d;
  rp.n = a.n;
  rp.co = a.co;
  // Between items every stage of the warp is free: each copy issued was
  // waited for and read before the previous item ended.
  int issued = ntiles < S ? ntiles : S;
  if (lane == 0)
    for (int j = 0; j < issued; ++j)
      issue_stage<KF>(a, stages + ((gt + j) % S) * kB, &full[(gt + j) % S], it.f_begin + j * KF);
  float2 ax[NP], ay[NP], az[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) ax[p] = ay[p] = az[p] = make_float2(0.f, 0.f);
  // The FP32 sums' rounding, more than the terms', sets the error, and the chained order
  // of a wake puts the large terms of a target next to one another. So a near sum spans
  // eight filaments before it joins the others, and these join the Kahan state after
  // each tile. Error against FP64 (2-norm) of a step of eight rotors: 4.7e-8 (Vatistas
  // core) and 4.2e-8 (cut-off) with one sum over 64 filaments, now 3.6e-8 and 3.3e-8, as
  // without chains, in input order (3.7e-8 and 3.3e-8). The sums take up to 3% longer for
  // it: 11.8 -> 11.9 ms on the large wake, 195 -> 199 us on 7.6k targets. (A second level
  // of sums, over 32, another fold between a tile's halves or two sets for the distant
  // form give 3.3e-8 to 3.5e-8 and cost 3 to 10%.)

  int i = 0;
  for (; i < ntiles; ++i) {
    const unsigned g = gt + i;
    const int st = g % S;
    const bool landed = mbar_wait_bounded(&full[st], (g / S) & 1u, a.err, a.wait_limit_ns);
    if (!__all_sync(0xffffffffu, landed)) break;
    unsigned char *stage = stages + st * kB;
    float4 *sP = reinterpret_cast<float4 *>(stage);  // KF records of 4
    // Filaments go in groups of 4; bit g of these masks is group g of the tile.
    // A warp-level screen (one filament per lane, every 32 filaments) sorts the
    // groups: all four filaments distant (above), core-free or not, and of the
    // others those near some target, whose near-singular bits (NearBits) go to
    // shared memory as one word for the FP64 pass. With the reach cut-off in
    // play every group is of the last kind.
    // Bit f of hm: filament f starts a chain (the sign of its |L|^2).
    unsigned careful = 0u, gfree = 0u, gdist = 0u;
    unsigned long long hm = 0;
    if (co_on) {
      careful = kGroups;
#pragma unroll 1
      for (int w = 0; w < KF / 32; ++w) {
        const int k = 32 * w + lane;
        const unsigned h = __ballot_sync(0xffffffffu, signbit(sP[4 * k + ((k >> 2) & 3)].w));
        hm |= (unsigned long long)h << (32 * w);
      }
    } else {
#pragma unroll 1
      for (int w = 0; w < KF / 32; ++w) {
        const int k = 32 * w + lane;
        float4 *r = sP + 4 * k;
        const int sw = (k >> 2) & 3;
        float4 A = r[0 ^ sw], B = r[1 ^ sw], C = r[2 ^ sw];
        const float4 D = r[3 ^ sw];
        // the warp's target ball (centre, radius, largest S2), kept in shared
        // memory so it holds no registers across the hot loops
        const float wcx = ws[0], wcy = ws[1], wcz = ws[2], wr = ws[3], rn_floor = ws[4];
        const float big = fabsf(wcx) + fabsf(wcy) + fabsf(wcz);
        const float L2 = fabsf(A.w);
        hm |= (unsigned long long)__ballot_sync(0xffffffffu, signbit(A.w)) << (32 * w);
        const float dx = (A.x - wcx) + C.x, dy = (A.y - wcy) + C.y, dz = (A.z - wcz) + C.z;
        const float mx = fmaf(0.5f, D.x, dx), my = fmaf(0.5f, D.y, dy), mz = fmaf(0.5f, D.z, dz);
        const float d2 = mx * mx + my * my + mz * mz;
        const float reach = sqrtf(fmaf(0.25f, L2, fmaxf(C.w, rn_floor)));
        const float slack =
            1e-5f * (big + fabsf(A.x) + fabsf(A.y) + fabsf(A.z)) + 1e-3f * (reach + wr);
        const float lim = wr + reach + slack;
        const bool far = d2 > lim * lim;
        // nearest approach of a warp target to the segment: its midpoint
        // distance less wr and |L|/2
        const float rmin = sqrtf(d2) - wr - 0.5f * sqrtf(L2) - slack;
        bool free_;
        if (MODEL == kCoreVatistas) {
          // distance of the ball centre from the filament's line: |L x (x1 - c)| / |L|;
          // every target of the warp is at least that less wr from it
          const float hx = D.y * dz - D.z * dy, hy = D.z * dx - D.x * dz, hz = D.x * dy - D.y * dx;
          const float h = sqrtf((hx * hx + hy * hy + hz * hz) / L2) - wr - slack;
          const float rc2 = B.w * B.w;
          // zero length: the pair term is zero on either form; rc = 0 (no core,
          // or K = 0 and a zero term): the factor is 1
          free_ = !(L2 > 0.f) || B.w == 0.f ||
                  (h > 0.f && h * h * h * fmaxf(h, rmin) >= kCoreFree4 * rc2 * rc2);
        } else {  // D.w = d |L|^2
          free_ = rmin > 0.f && rmin * rmin >= kCutoffFreeSq * sqrtf(D.w);
        }
        // both endpoints kDistantRatio ball radii from the centre, all in range
        const float q1 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        const float ex = dx + D.x, ey = dy + D.y, ez = dz + D.z;
        const float q2 = ex * ex + ey * ey + ez * ez;
        const float dmin = fmaxf(kDistantRatio * kDistantRatio * wr * wr, kDistantMinSq);
        const float qmax = fmaxf(q1, q2);
        const bool dist = far && fminf(q1, q2) >= dmin && qmax <= kDistantMaxSq;
        const bool cored = qmax * (B.x * B.x + B.y * B.y + B.z * B.z) <= kDistantMaxMq;
        careful |= nibble_any(__ballot_sync(0xffffffffu, !far)) << (8 * w);
        const unsigned gf = nibble_all(__ballot_sync(0xffffffffu, free_ && far));
        const unsigned gd = nibble_all(__ballot_sync(0xffffffffu, dist)) &
                            (gf | nibble_all(__ballot_sync(0xffffffffu, cored)));
        free_cnt += 4u * live_slots * __popc(gd & gf);
        gfree |= (gd & gf) << (8 * w);
        gdist |= gd << (8 * w);
        if ((gd >> (lane >> 2)) & 1u) {
          const float nx = 2.f * B.x, ny = 2.f * B.y, nz = 2.f * B.z;
          r[0 ^ sw] = make_float4(dx, dy, dz, q1);
          r[2 ^ sw] = make_float4(dy * nz - dz * ny, dz * nx - dx * nz, dx * ny - dy * nx, 0.f);
          if (MODEL == kCoreVatistas && !((gf >> (lane >> 2)) & 1u)) {
            r[1 ^ sw] = make_float4(B.x, B.y, B.z, -L2);
            r[3 ^ sw] = make_float4(D.x, D.y, D.z, 16.f * D.w);
          } else {
            r[1 ^ sw] = make_float4(nx, ny, nz, -L2);
            r[3 ^ sw] = make_float4(D.x, D.y, D.z, 2.f * D.w);
          }
        }
      }
      __syncwarp();
    }
    // the first filament after a group of another form starts a chain too
    const auto group_heads = [&](int gr) { return (unsigned)(hm >> (4 * gr)) & 15u; };
    if (gdist) {
      float2 mx[NP], my[NP], mz[NP], p2[NP], Ax[NP], Ay[NP], Az[NP], ti[NP], tr[NP];
      const float ox = cx - ws[0], oy = cy - ws[1], oz = cz - ws[2];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const float2 x = make_float2(s_p[2 * p * 32 + lane] + ox, s_p[(2 * p + 1) * 32 + lane] + ox);
        const float2 y = make_float2(s_p[(T + 2 * p) * 32 + lane] + oy,
                                     s_p[(T + 2 * p + 1) * 32 + lane] + oy);
        const float2 z = make_float2(s_p[(2 * T + 2 * p) * 32 + lane] + oz,
                                     s_p[(2 * T + 2 * p + 1) * 32 + lane] + oz);
        p2[p] = __ffma2_rn(x, x, __ffma2_rn(y, y, __fmul2_rn(z, z)));
        mx[p] = __fmul2_rn(bc(-2.f), x);
        my[p] = __fmul2_rn(bc(-2.f), y);
        mz[p] = __fmul2_rn(bc(-2.f), z);
        Ax[p] = Ay[p] = Az[p] = make_float2(0.f, 0.f);
      }
      // Tiles of 32 filaments that all start a chain (a set without connected filaments)
      // have a loop of their own for the core-free groups: 60k random filaments onto 60k
      // targets 3.94 ms (Vatistas) and 3.61 (cut-off), through the loop below 4.41 and
      // 4.37. Tiles of 64, the faster ones on wakes, do without: with it the large wake's
      // sum takes 12.2 ms instead of 11.9. The autotuner times both on each set.
      const unsigned alone = KF == 32 && (unsigned)hm == 0xffffffffu ? gfree : 0u;
#pragma unroll 1
      for (unsigned gm = alone; gm; gm &= gm - 1u) {
        const int gr = __ffs(gm) - 1, sw = gr & 3;
        const float4 *rec = sP + 16 * gr;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 qa = rec[4 * j + (0 ^ sw)];
          distant_start<NP>(qa, rec[4 * j + (3 ^ sw)], mx, my, mz, p2, ti, tr);
          distant_filament<NP, kNoCore>(qa, rec[4 * j + (1 ^ sw)], rec[4 * j + (2 ^ sw)], 0.f, mx,
                                        my, mz, p2, ax, ay, az, Ax, Ay, Az, ti, tr);
        }
      }
      int last = -2;
#pragma unroll 1
      for (unsigned gm = gdist & ~alone; gm; gm &= gm - 1u) {
        const int gr = __ffs(gm) - 1;
        const unsigned hg = group_heads(gr) | (gr != last + 1 ? 1u : 0u);
        last = gr;
        const float4 *rec = sP + 16 * gr;
        const int sw = gr & 3;
        if (hg & 1u) distant_start<NP>(rec[0 ^ sw], rec[3 ^ sw], mx, my, mz, p2, ti, tr);
        if (((gfree >> gr) & 1u) && !(hg & 14u)) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            distant_filament<NP, kNoCore>(rec[4 * j + (0 ^ sw)], rec[4 * j + (1 ^ sw)],
                                          rec[4 * j + (2 ^ sw)], 0.f, mx, my, mz, p2, ax, ay, az,
                                          Ax, Ay, Az, ti, tr);
        } else {
          const bool core = !((gfree >> gr) & 1u);
#pragma unroll 1
          for (int j = 0; j < 4; ++j) {
            const float4 qa = rec[4 * j + (0 ^ sw)], qd = rec[4 * j + (3 ^ sw)];
            const float4 qb = rec[4 * j + (1 ^ sw)], qc = rec[4 * j + (2 ^ sw)];
            if (j > 0 && ((hg >> j) & 1u)) distant_start<NP>(qa, qd, mx, my, mz, p2, ti, tr);
            if (MODEL == kCoreCutoff || core)
              distant_filament<NP, MODEL>(qa, qb, qc, qd.w, mx, my, mz, p2, ax, ay, az, Ax, Ay, Az,
                                          ti, tr);
            else
              distant_filament<NP, kNoCore>(qa, qb, qc, 0.f, mx, my, mz, p2, ax, ay, az, Ax, Ay, Az,
                                            ti, tr);
          }
        }
      }
#pragma unroll
      for (int p = 0; p < NP; ++p) {  // - p x A
        ax[p] = __ffma2_rn(bc(0.5f), __ffma2_rn(my[p], Az[p], neg2(__fmul2_rn(mz[p], Ay[p]))), ax[p]);
        ay[p] = __ffma2_rn(bc(0.5f), __ffma2_rn(mz[p], Ax[p], neg2(__fmul2_rn(mx[p], Az[p]))), ay[p]);
        az[p] = __ffma2_rn(bc(0.5f), __ffma2_rn(mx[p], Ay[p], neg2(__fmul2_rn(my[p], Ax[p]))), az[p]);
      }
    }
    unsigned mine = 0u;  // this lane's groups with near-singular pairs
    if (gdist != kGroups) {
      float2 npx[NP], npy[NP], npz[NP], ti[NP];  // -(P - c)
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        npx[p] = make_float2(-s_p[2 * p * 32 + lane], -s_p[(2 * p + 1) * 32 + lane]);
        npy[p] = make_float2(-s_p[(T + 2 * p) * 32 + lane], -s_p[(T + 2 * p + 1) * 32 + lane]);
        npz[p] = make_float2(-s_p[(2 * T + 2 * p) * 32 + lane],
                             -s_p[(2 * T + 2 * p + 1) * 32 + lane]);
        ti[p] = make_float2(0.f, 0.f);
      }
      float2 gx[NP], gy[NP], gz[NP];  // over eight filaments
#pragma unroll
      for (int p = 0; p < NP; ++p) gx[p] = gy[p] = gz[p] = make_float2(0.f, 0.f);
      int last = -2;
#pragma unroll 1
      for (unsigned gm = ~gdist & kGroups; gm; gm &= gm - 1u) {
        const int gr = __ffs(gm) - 1;
        const unsigned hg = group_heads(gr) | (gr != last + 1 ? 1u : 0u);
        last = gr;
        const bool near_some = (careful >> gr) & 1u;
        const float4 *rec = sP + 16 * gr;
        unsigned nbits = 0;
#pragma unroll 2
        for (int j = 0; j < 4; ++j) {
          const Fil f = load_filament(rec + 4 * j, gr & 3, cx, cy, cz);
          // near-singular threshold, raised for threads whose targets spread far
          // from their centre (the FP32 differences lose ~eps * spread / |r1|)
          const float Rn2 = fmaxf(f.Rn2, S2);
          if ((hg >> j) & 1u) chain_start<NP>(f, npx, npy, npz, ti);
          unsigned m = 0;
#pragma unroll
          for (int p = 0; p < NP; ++p)
            interact<MODEL>(npx[p], npy[p], npz[p], f, Rn2, near_some, co2, co_on, gx[p], gy[p],
                            gz[p], m, 1u << (2 * p), 2u << (2 * p), ti[p]);
          nbits |= m << (kPer * j);
        }
        if ((gr & 1) || gm < (2u << gr)) {  // the second of a pair of groups, or the last
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            ax[p] = __fadd2_rn(ax[p], gx[p]);
            ay[p] = __fadd2_rn(ay[p], gy[p]);
            az[p] = __fadd2_rn(az[p], gz[p]);
            gx[p] = gy[p] = gz[p] = make_float2(0.f, 0.f);
          }
        }
        if (near_some) {
          s_nb[gr * 32 + lane] = (typename NearBits<T>::type)nbits;
          if (nbits) mine |= 1u << gr;
        }
      }
    }
    __syncwarp();
    // into the Kahan state
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const int sl = lane * T + 2 * p;
      kahan_add(s_k[0 * 32 * T + sl], s_k[1 * 32 * T + sl], ax[p].x);
      kahan_add(s_k[2 * 32 * T + sl], s_k[3 * 32 * T + sl], ay[p].x);
      kahan_add(s_k[4 * 32 * T + sl], s_k[5 * 32 * T + sl], az[p].x);
      kahan_add(s_k[0 * 32 * T + sl + 1], s_k[1 * 32 * T + sl + 1], ax[p].y);
      kahan_add(s_k[2 * 32 * T + sl + 1], s_k[3 * 32 * T + sl + 1], ay[p].y);
      kahan_add(s_k[4 * 32 * T + sl + 1], s_k[5 * 32 * T + sl + 1], az[p].y);
      ax[p] = ay[p] = az[p] = make_float2(0.f, 0.f);
    }
    // Near-singular pairs of this tile: the reference formula in FP64, added to
    // the owner's Kahan state as an exact hi + lo pair. In rounds, every lane
    // lists the next kList of its pairs in the consumed stage (its groups in
    // order, so every target receives its terms in the order of the filaments),
    // all lanes compute the list together, and each adds its own. (With the
    // pairs listed lane by lane, few lanes wrote at a time and each list was
    // scanned for from the start: half of the time of the warps that bound a
    // small wake, 149k of 312k cycles for a tile range with 792 pairs.)
    if (careful) {  // warp-uniform
      constexpr int kList = kB / (int)sizeof(NearEntry) / 32;
      NearEntry *ne = reinterpret_cast<NearEntry *>(stages + st * kB);
      unsigned bits = 0u, w = 0u;
#pragma unroll 1
      while (__any_sync(0xffffffffu, (bits | mine) != 0u)) {
        int at[kList], n = 0;
#pragma unroll
        for (int r = 0; r < kList; ++r) {
          if (!bits && mine) {
            w = __ffs(mine) - 1;
            mine &= mine - 1u;
            bits = s_nb[w * 32 + lane];
          }
          const unsigned m = __ballot_sync(0xffffffffu, bits != 0u);
          at[r] = -1;
          if (bits) {
            const int b = __ffs(bits) - 1;
            bits &= bits - 1u;
            at[r] = n + __popc(m & ((1u << lane) - 1u));
            ne[at[r]].fidx = it.f_begin + i * KF + 4 * w + b / kPer;
            ne[at[r]].slot = lane * T + b % kPer;
            ++near_cnt;
          }
          n += __popc(m);
        }
        __syncwarp();
        for (int k = lane; k < n; k += 32) {
          NearEntry &e = ne[k];
          int local = e.slot;
          if (local >= tl.t_count) local = tl.t_count - 1;
          const double4 p = a.tp[tl.t_begin + local];
          double u0 = 0.0, u1 = 0.0, u2 = 0.0;
          pair64(a.ra[e.fidx], a.rb[e.fidx], p.x, p.y, p.z, rp, u0, u1, u2);
          e.u[0] = u0;
          e.u[1] = u1;
          e.u[2] = u2;
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kList; ++r) {
          if (at[r] < 0) continue;
          const NearEntry &e = ne[at[r]];
          const int sl = e.slot;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const float hi = (float)e.u[c];
            const float lo = (float)(e.u[c] - (double)hi);
            kahan_add(s_k[(2 * c) * 32 * T + sl], s_k[(2 * c + 1) * 32 * T + sl], hi);
            kahan_add(s_k[(2 * c) * 32 * T + sl], s_k[(2 * c + 1) * 32 * T + sl], lo);
          }
        }
        __syncwarp();
      }
    }
    // Every lane is done with the stage (tile and near list). Lanes wrote to it
    // (prepared records, near list): each orders its own accesses before the copy
    // that fills it next, tile i + S here or a tile of the warp's next item.
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0 && issued < ntiles) {
      issue_stage<KF>(a, stages + st * kB, &full[st], it.f_begin + issued * KF);
    }
    if (issued < ntiles) ++issued;
    __syncwarp();
  }
  if (i < ntiles) {
    // A bounded wait ran out: let the copies already issued land (bounded)
    // before the warp leaves, so no bulk copy targets the shared memory of a
    // finished CTA.
    if (lane == 0)
      for (int j = i; j < issued; ++j) {
        const unsigned g = gt + j;
        mbar_wait_bounded(&full[g % S], (g / S) & 1u, a.err, a.wait_limit_ns);
      }
    __syncwarp();
    return false;
  }
  gt += ntiles;
  return true;
}

// Resident CTAs per SM the register allocation is capped for. The loops want
// registers for four filaments in flight more than they want warps: with six
// targets a lane, 3 CTAs (168 registers) run the large wake at 1289 Gint/s, 4
// CTAs (128, spills) at 1159, 2 CTAs at 1184; with four targets 4 CTAs run the
// 60k-filament cut-off wake at 1193, 3 at 1148, 5 at 1072.
template <int T>
struct MinBlocks {
  static constexpr int value = T <= 2 ? 5 : (T == 4 ? 4 : (T == 6 ? 3 : 2));
};

template <int T, int KF, int MODEL>
__global__ void __launch_bounds__(kThreads, MinBlocks<T>::value) bs_f32c(const F32cArgs a) {
  after_previous();
  static_assert(KF % 32 == 0 && KF <= 64, "one screen word per 32 filaments, a head bit per filament");
  static_assert(T % 2 == 0 && T <= 8, "targets go in pairs, near-singular bits eight to a filament");
  constexpr int S = StageSmem<KF>::kStages;
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  unsigned char *stages = smem + (threadIdx.x >> 5) * warp_smem_bytes<T, KF>();
  float *s_k = reinterpret_cast<float *>(stages + S * StageSmem<KF>::kBytes);
  float *s_p = s_k + 6 * 32 * T;
  auto *s_nb = reinterpret_cast<typename NearBits<T>::type *>(s_p + 3 * 32 * T);
  uint64_t *full = reinterpret_cast<uint64_t *>(s_nb + (KF / 4) * 32);
  float *ws = reinterpret_cast<float *>(full + S);
  if (lane == 0) {
    for (int st = 0; st < S; ++st) mbar_init(&full[st], 1);
    fence_mbar_init();
  }
  __syncwarp();
  const bool co_on = co_can_trigger(a.bbox, a.co);
  unsigned gt = 0;
  unsigned near_cnt = 0;
  unsigned long long free_cnt = 0;  // pairs of this lane that took the core-free form
  while (true) {
    int q = 0;
    if (lane == 0) q = (int)atomicAdd(a.work_ctr, 1u);
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q >= a.n_items) break;
    const int item_id = a.order ? a.order[q] : q;
    Item it = a.items[item_id];
    Tile tl = a.tiles[it.tile];
    if (a.live && !clip_live(a.live, it, tl)) continue;
    if (tl.t_count <= 0 || ((it.f_end - it.f_begin) % KF) != 0) {
      if (lane == 0) atomicOr(a.err, kErrBadItem);
      continue;
    }
    // This lane's T consecutive targets, relative to the FP32 image of the first.
    float px[T], py[T], pz[T];
    float spread2 = 0.f;
    int l0 = lane * T;
    if (l0 >= tl.t_count) l0 = tl.t_count - 1;
    const double4 p0 = a.tp[tl.t_begin + l0];
    const float cx = (float)p0.x, cy = (float)p0.y, cz = (float)p0.z;
#pragma unroll
    for (int t = 0; t < T; ++t) {
      int l = lane * T + t;
      if (l >= tl.t_count) l = tl.t_count - 1;
      const double4 p = a.tp[tl.t_begin + l];
      px[t] = (float)(p.x - (double)cx);
      py[t] = (float)(p.y - (double)cy);
      pz[t] = (float)(p.z - (double)cz);
      spread2 = fmaxf(spread2, px[t] * px[t] + py[t] * py[t] + pz[t] * pz[t]);
      s_p[t * 32 + lane] = px[t];
      s_p[(T + t) * 32 + lane] = py[t];
      s_p[(2 * T + t) * 32 + lane] = pz[t];
#pragma unroll
      for (int c = 0; c < 6; ++c) s_k[c * 32 * T + lane * T + t] = 0.f;
    }
    const float S2 = 0.09f * spread2;  // pairs closer than 0.3 x spread go to FP64
    // The warp's targets lie in the ball (wc, wr) around the centre of their
    // bounding box. As r1.r2 = |P - m|^2 - |L|^2/4 (m the filament midpoint),
    // a filament whose midpoint is farther than wr + sqrt(|L|^2/4 + Rn^2)
    // from wc has r1.r2 >= Rn^2 for every target of the warp; rn_floor is
    // the warp's largest per-thread threshold S2.
    float blo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, bhi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const float q[3] = {cx + px[t], cy + py[t], cz + pz[t]};
#pragma unroll
      for (int c = 0; c < 3; ++c) blo[c] = fminf(blo[c], q[c]), bhi[c] = fmaxf(bhi[c], q[c]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        blo[c] = fminf(blo[c], __shfl_xor_sync(0xffffffffu, blo[c], o));
        bhi[c] = fmaxf(bhi[c], __shfl_xor_sync(0xffffffffu, bhi[c], o));
      }
    const float wcx = 0.5f * (blo[0] + bhi[0]);
    const float wcy = 0.5f * (blo[1] + bhi[1]);
    const float wcz = 0.5f * (blo[2] + bhi[2]);
    float wr2 = 0.f;
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const float dx = (cx - wcx) + px[t], dy = (cy - wcy) + py[t], dz = (cz - wcz) + pz[t];
      wr2 = fmaxf(wr2, dx * dx + dy * dy + dz * dz);
    }
    float rn_floor = S2;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      wr2 = fmaxf(wr2, __shfl_xor_sync(0xffffffffu, wr2, o));
      rn_floor = fmaxf(rn_floor, __shfl_xor_sync(0xffffffffu, rn_floor, o));
    }
    if (lane == 0) {
      ws[0] = wcx;
      ws[1] = wcy;
      ws[2] = wcz;
      ws[3] = sqrtf(wr2);
      ws[4] = rn_floor;
    }
    __syncwarp();
    const bool ok = f32c_item<T, KF, MODEL>(a, it, stages, full, s_k, s_p, s_nb, gt, cx, cy, cz, S2,
                                            ws, co_on, near_cnt, free_cnt, tl);
    if (!ok) break;
    double *part = a.part + (size_t)item_id * 3 * a.tile_cap;
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const int l = lane * T + t;
      if (l < tl.t_count) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
          part[c * a.tile_cap + l] = (double)s_k[(2 * c) * 32 * T + l] -
                                     (double)s_k[(2 * c + 1) * 32 * T + l];
      }
    }
    __syncwarp();
  }
  if (a.near_ctr && near_cnt) atomicAdd(a.near_ctr, (unsigned long long)near_cnt);
  if (a.near_ctr && free_cnt) atomicAdd(a.near_ctr + 1, free_cnt);
}

// ------------------------------------------------------- FP64 direct sum
constexpr int kF64Threads = 128;
constexpr int kF64Tile = 64;  // filaments per shared-memory stage

// A thread per target, filaments through shared memory. FORM kF64Ref: ref_pair's
// terms added in order, what a sequential evaluation promises and a general
// Vatistas index needs; otherwise the short form of the core model, with ref_pair
// for the pairs that it leaves. Bound by the FP64 units (69% of their cycles, 56
// operations a pair, where ref_pair's three roots and four divisions make some
// 150): 12.5k targets x 24.7k filaments take 1.46 ms, 3.03 with ref_pair
// throughout (cut-off core 1.11, 1.86). Two targets a thread take 1.76 ms, 40
// registers less 1.48.
enum F64Form : int { kF64Ref = 0, kF64Vatistas = 1, kF64Cutoff = 2 };
static F64Form f64_form(int model, double n, bool sequential) {
  if (sequential || (model != kCoreCutoff && n != 2.0)) return kF64Ref;
  return model == kCoreCutoff ? kF64Cutoff : kF64Vatistas;
}

template <int FORM>
__global__ void __launch_bounds__(kF64Threads) bs_f64(const F32cArgs a) {
  after_previous();
  constexpr bool kShort = FORM != kF64Ref;
  constexpr int kModel = FORM == kF64Cutoff ? kCoreCutoff : kCoreVatistas;
  __shared__ double4 sA[2][kF64Tile], sB[2][kF64Tile], sC[kShort ? 2 : 1][kShort ? kF64Tile : 1];
  __shared__ int sD[kShort ? 2 : 1][kShort ? kF64Tile : 1];
  __shared__ int s_item;
  const int tid = threadIdx.x;
  RefParams rp;
  rp.model = a.model;
  rp.d = a.d;
  rp.n = a.n;
  rp.co = a.co;
  const int co_hi = reach_hi(a.co);
  const auto stage = [&](int b, const double4 A, const double4 B) {
    sA[b][tid] = A;
    sB[b][tid] = B;
    if constexpr (kShort) {
      const double x = B.x - A.x, y = B.y - A.y, z = B.z - A.z, L2 = fma(x, x, fma(y, y, z * z));
      double w = FORM == kF64Cutoff ? a.d * L2 : B.w * L2;
      if (FORM == kF64Vatistas) w *= w;
      if (!isfinite(A.w)) w = NAN;  // such a filament adds nothing: left to ref_pair
      sC[b][tid] = make_double4(x, y, z, w);
      sD[b][tid] = axis_limit(L2);
    }
  };
  while (true) {
    if (tid == 0) s_item = (int)atomicAdd(a.work_ctr, 1u);
    __syncthreads();
    const int q = s_item;
    __syncthreads();
    if (q >= a.n_items) break;
    const int item_id = a.order ? a.order[q] : q;
    Item it = a.items[item_id];
    Tile tl = a.tiles[it.tile];
    if (a.live && !clip_live(a.live, it, tl)) continue;  // uniform over the block
    const double4 p = a.tp[tl.t_begin + (tid < tl.t_count ? tid : tl.t_count - 1)];
    double u[3] = {0.0, 0.0, 0.0}, v[3] = {0.0, 0.0, 0.0};
    const int ntiles = (it.f_end - it.f_begin) / kF64Tile;
    if (tid < kF64Tile) stage(0, a.ra[it.f_begin + tid], a.rb[it.f_begin + tid]);
    __syncthreads();
    for (int i = 0; i < ntiles; ++i) {
      const int b = i & 1;
      double4 nA, nB;
      const bool more = i + 1 < ntiles && tid < kF64Tile;
      if (more) {
        nA = a.ra[it.f_begin + (i + 1) * kF64Tile + tid];
        nB = a.rb[it.f_begin + (i + 1) * kF64Tile + tid];
      }
#pragma unroll 1
      for (int k = 0; k < kF64Tile; ++k) {
        const double4 A = sA[b][k], B = sB[b][k];
        if constexpr (kShort) {
          if (!pair64_short<kModel>(A, B, sC[b][k], sD[b][k], p.x, p.y, p.z, co_hi, v[0], v[1], v[2]))
            ref_pair<false>(A, B, p.x, p.y, p.z, rp, u[0], u[1], u[2]);
        } else {
          ref_pair(A, B, p.x, p.y, p.z, rp, u[0], u[1], u[2]);
        }
      }
      if (more) stage(b ^ 1, nA, nB);
      __syncthreads();
    }
    if (tid < tl.t_count) {
      double *part = a.part + (size_t)item_id * 3 * a.tile_cap + tid;
#pragma unroll
      for (int c = 0; c < 3; ++c)
        part[c * a.tile_cap] = kShort ? fma(v[c], 1.0 / k4Pi, u[c]) : u[c];
    }
  }
}

// --------------------------------------------------------------- reduce
// A block sums 32 consecutive targets of a tile: each warp a run of the tile's
// items in order, lanes the targets, then the warps' sums in order. (One thread
// per target, all items in one chain of loads, took 30 us on the 3.1k-target
// wake; spread over eight warps 12.) With a live table, only the live targets of a
// tile are written, from the items before the group's live filament end (a tile's
// items cover increasing filament ranges, so those come first). The last kernel of
// an evaluation: it leaves the work queue at its start.
constexpr int kReduceWarps = 8;
__global__ void __launch_bounds__(32 * kReduceWarps)
    bs_reduce(const Tile *__restrict__ tiles, const Group *__restrict__ groups,
              const double *__restrict__ part, const int *__restrict__ perm, int tile_cap,
              const Item *__restrict__ items, const GroupLive *__restrict__ live, unsigned *ctr) {
  after_previous();
  __shared__ double s_sum[kReduceWarps][3][32];
  if (blockIdx.x + blockIdx.y == 0 && threadIdx.x == 0) *ctr = 0u;
  Tile tl = tiles[blockIdx.x];
  const Group g = groups[tl.group];
  if (live) {
    const GroupLive gl = live[tl.group];
    const long long tn = gl.t_end - tl.t_begin;
    if (tn <= 0) return;
    if (tn < tl.t_count) tl.t_count = (int)tn;
    int lo = 0, hi = tl.n_items;  // the first item at or past the live end
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (items[tl.first_item + mid].f_begin < gl.f_end) lo = mid + 1; else hi = mid;
    }
    tl.n_items = lo;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int l = 32 * blockIdx.y + lane;
  if (32 * (int)blockIdx.y >= tl.t_count) return;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0;
  if (l < tl.t_count) {
    const int k0 = tl.n_items * warp / kReduceWarps, k1 = tl.n_items * (warp + 1) / kReduceWarps;
    const double *p = part + (size_t)(tl.first_item + k0) * 3 * tile_cap + l;
#pragma unroll 4
    for (int k = k0; k < k1; ++k, p += 3 * (size_t)tile_cap) {
      s0 += p[0];
      s1 += p[tile_cap];
      s2 += p[2 * tile_cap];
    }
  }
  s_sum[warp][0][lane] = s0, s_sum[warp][1][lane] = s1, s_sum[warp][2][lane] = s2;
  __syncthreads();
  if (warp >= 3 || l >= tl.t_count) return;
  double s = 0.0;  // warp c: component c
#pragma unroll
  for (int w = 0; w < kReduceWarps; ++w) s += s_sum[w][warp][lane];
  const long long local = (long long)perm[tl.t_begin + l] - g.t_begin;
  const long long j = local / g.ns_p, i = local - j * g.ns_p;
  double *o = g.out + i + 3 * g.ns_p * j + warp * g.ns_p;
  *o = g.accumulate ? *o + s : s;
}

// --------------------------------------------------------------- lengths
__global__ void bs_length(const double *__restrict__ F1, const double *__restrict__ F2,
                          long long d0, long long nf, double *L) {
  const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  const long long j = f / d0, i = f - j * d0;
  const long long b = i + d0 * 3 * j;
  const double dx = F2[b] - F1[b], dy = F2[b + d0] - F1[b + d0], dz = F2[b + 2 * d0] - F1[b + 2 * d0];
  L[f] = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
}

// ------------------------------------------------------- FP32 FMA peak probe
// Each thread runs 8 independent FMA chains; nothing but FFMA issues in the
// loop body, so the rate is the FP32 pipe's (the direct sum's roofline).
__global__ void __launch_bounds__(256) bs_ffma_peak(float *out, int iters, float a, float b) {
  float x0 = threadIdx.x * 1e-7f, x1 = x0 + 1e-3f, x2 = x0 + 2e-3f, x3 = x0 + 3e-3f;
  float x4 = x0 + 4e-3f, x5 = x0 + 5e-3f, x6 = x0 + 6e-3f, x7 = x0 + 7e-3f;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      x0 = fmaf(x0, a, b);
      x1 = fmaf(x1, a, b);
      x2 = fmaf(x2, a, b);
      x3 = fmaf(x3, a, b);
      x4 = fmaf(x4, a, b);
      x5 = fmaf(x5, a, b);
      x6 = fmaf(x6, a, b);
      x7 = fmaf(x7, a, b);
    }
  }
  const float r = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
  if (r == 12345.678f) out[blockIdx.x * blockDim.x + threadIdx.x] = r;  // keeps the chains live
}

// ------------------------------------------------------- bounded-wait self-test
// Waits on an mbarrier that nothing arrives on, with the given limit; the
// bounded wait must give up, set the error word and let the kernel return.
__global__ void bs_wait_selftest(unsigned *err, unsigned long long limit_ns) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_wait_bounded(&bar, 0u, err, limit_ns);
  __syncthreads();
}

__global__ void bs_roots_selftest(const double *__restrict__ x, long long n, double *y) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  y[i] = rsqrt64(x[i]);
  y[n + i] = rcp64(x[i]);
  y[2 * n + i] = rsqrt(x[i]);
  y[3 * n + i] = 1.0 / x[i];
}

// ============================================================ host launchers
namespace {
template <int T, int KF, int MODEL>
cudaError_t launch_f32c_t(const F32cArgs &a, int grid, cudaStream_t s) {
  const size_t smem = f32c_smem_bytes_t<T, KF>();
  static unsigned attr_set = 0;  // one bit per device: the attribute is per context
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 32 || !(attr_set & (1u << dev))) {
    cudaError_t e = cudaFuncSetAttribute(bs_f32c<T, KF, MODEL>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(bs_f32c<T, KF, MODEL>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    if (dev < 32) attr_set |= (1u << dev);
  }
  // `grid` counts workers (warps); kWarps of them per CTA
  bs_f32c<T, KF, MODEL><<<(grid + kWarps - 1) / kWarps, kThreads, smem, s>>>(a);
  return cudaGetLastError();
}

template <int T, int KF, int MODEL>
int occupancy_t() {
  const size_t smem = f32c_smem_bytes_t<T, KF>();
  cudaFuncSetAttribute(bs_f32c<T, KF, MODEL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)smem);
  cudaFuncSetAttribute(bs_f32c<T, KF, MODEL>, cudaFuncAttributePreferredSharedMemoryCarveout,
                       (int)cudaSharedmemCarveoutMaxShared);
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, bs_f32c<T, KF, MODEL>, kThreads, smem) !=
      cudaSuccess)
    return kWarps;
  return (n > 0 ? n : 1) * kWarps;  // resident workers per SM
}

#define WINDS_F32C_CASE(FN, M, TT, KK, ...) \
  case M * 1000 + TT * 100 + KK / 32: return FN<TT, KK, M>(__VA_ARGS__);
#define WINDS_F32C_KF(FN, M, TT, ...) \
  WINDS_F32C_CASE(FN, M, TT, 32, __VA_ARGS__) WINDS_F32C_CASE(FN, M, TT, 64, __VA_ARGS__)
#define WINDS_F32C_T(FN, M, ...)                                              \
  WINDS_F32C_KF(FN, M, 2, __VA_ARGS__) WINDS_F32C_KF(FN, M, 4, __VA_ARGS__) \
  WINDS_F32C_KF(FN, M, 6, __VA_ARGS__) WINDS_F32C_KF(FN, M, 8, __VA_ARGS__)
#define WINDS_F32C_DISPATCH(FN, ...)                                           \
  switch (model * 1000 + f32c_targets(T) * 100 + (KF < 64 ? KF : 64) / 32) {  \
    WINDS_F32C_T(FN, 0, __VA_ARGS__) WINDS_F32C_T(FN, 1, __VA_ARGS__) default: break; \
  }
}  // namespace

bool f32c_config_supported(int T, int KF) {
  return (T == 2 || T == 3 || T == 4 || T == 8) && (KF == 32 || KF == 64 || KF == 128);
}

// Targets per lane of a choice: they go in pairs, T = 3 (three pairs) runs with
// six. KF = 128 runs as 64.
int f32c_targets(int T) { return T == 3 ? 6 : T; }
int f32c_tile(int T) { return 32 * f32c_targets(T); }
int f32c_quantum(int KF) { return KF < 64 ? KF : 64; }
int f32c_warps() { return kWarps; }
int f64_threads() { return kF64Threads; }
int f64_tile() { return kF64Tile; }

cudaError_t launch_f32c(const F32cArgs &a, int model, int T, int KF, int grid, cudaStream_t s) {
  WINDS_F32C_DISPATCH(launch_f32c_t, a, grid, s)
  return cudaErrorInvalidValue;
}

int f32c_occupancy(int model, int T, int KF) {
  WINDS_F32C_DISPATCH(occupancy_t)
  return 1;
}

using F64Kernel = void (*)(const F32cArgs);
static F64Kernel f64_kernel(int model, double n, bool sequential) {
  const F64Form f = f64_form(model, n, sequential);
  return f == kF64Ref ? bs_f64<kF64Ref> : f == kF64Cutoff ? bs_f64<kF64Cutoff> : bs_f64<kF64Vatistas>;
}

int f64_occupancy(int model, double n, bool sequential) {
  int k = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, f64_kernel(model, n, sequential), kF64Threads,
                                                    0) != cudaSuccess)
    return 1;
  return k > 0 ? k : 1;
}

cudaError_t launch_f64(const F32cArgs &a, bool sequential, int grid, cudaStream_t s) {
  f64_kernel(a.model, a.n, sequential)<<<grid, kF64Threads, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_begin(BBox *bb, unsigned *ctr, unsigned long long *near, unsigned long long *cnt,
                         cudaStream_t s) {
  launch_after(bs_begin, 1, 32, 0, s, bb, ctr, near, cnt);
  return cudaGetLastError();
}

cudaError_t launch_pack(const winds_bs_family *fams, int nfam, unsigned long long *cnt,
                        long long pad_to, int model, double dcut, const PackedFilaments &pf,
                        const double *P, long long ns, long long nt, const TargetBufs &tb, BBox *bb,
                        cudaStream_t s, int *launches) {
  const int bs = 256;
  long long off = 0;
  int k = 0;
  bool first = true;
  do {
    PackArgs a;
    a.nfam = 0;
    long long blocks = 0;
    for (; k < nfam && a.nfam < kPackFams; ++k) {
      const winds_bs_family &m = fams[k];
      const long long nf = m.dims[0] * m.dims[2] * m.dims[3];
      if (nf <= 0) continue;
      PackArgs::Fam &f = a.fam[a.nfam];
      f.F1 = m.F1, f.F2 = m.F2, f.gam = m.gamma, f.rc = m.rc;
      f.d0 = m.dims[0], f.d2 = m.dims[2], f.nf = nf, f.off = off;
      f.cnt = cnt ? cnt + 2 * a.nfam : nullptr;
      ++a.nfam;
      f.block0 = (int)blocks;
      blocks += (nf + bs - 1) / bs;
      off += nf;
    }
    const bool last = k >= nfam;
    a.model = model, a.dcut = dcut;
    a.pk = pf.pk, a.ra = pf.ra, a.rb = pf.rb, a.bb = bb;
    a.P = P, a.ns = ns, a.nt = last ? nt : 0;
    a.tp_raw = tb.tp_raw, a.tgroup = tb.tgroup;
    a.pad_block0 = (int)blocks;
    a.pad_from = off;
    a.pad_to = last ? pad_to : off;
    if (cnt && blocks > 0) {
      if (!first) {
        const cudaError_t e = cudaMemsetAsync(cnt, 0, 2 * kPackFams * sizeof(*cnt), s);
        if (e != cudaSuccess) return e;
      }
      first = false;
      launch_after(bs_chain_count, (unsigned)blocks, bs, 0, s, a);
      if (launches) ++*launches;
    }
    blocks += (a.pad_to - a.pad_from + bs - 1) / bs;
    a.tgt_block0 = (int)blocks;
    blocks += (a.nt + bs - 1) / bs;
    if (blocks > 0) {
      launch_after(bs_pack, (unsigned)blocks, bs, 0, s, a);
      if (launches) ++*launches;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  } while (k < nfam);
  return cudaSuccess;
}

cudaError_t launch_gather_targets(const double4 *src, const int *perm, long long n, double4 *dst,
                                  cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  launch_after(bs_gather_targets, (unsigned)((n + 255) / 256), 256, 0, s, src, perm, n, dst);
  return cudaGetLastError();
}

// The device-wide sort: 31-bit keys for one group, the group id above them for
// more, and only these bits sorted (one group: four passes of the library's
// radix sort, where all 64 bits took eight).
static int group_bits(int groups) {
  int b = 0;
  while ((1ll << b) < groups) ++b;
  return b;
}

cudaError_t sort_targets_bytes(long long n, int groups, size_t *bytes) {
  *bytes = 0;
  if (groups == 1)
    return cub::DeviceRadixSort::SortPairs(nullptr, *bytes, (const unsigned *)nullptr,
                                           (unsigned *)nullptr, (const int *)nullptr,
                                           (int *)nullptr, (int)n, 0, 31, (cudaStream_t)0);
  return cub::DeviceRadixSort::SortPairs(nullptr, *bytes, (const unsigned long long *)nullptr,
                                         (unsigned long long *)nullptr, (const int *)nullptr,
                                         (int *)nullptr, (int)n, 0, 31 + group_bits(groups),
                                         (cudaStream_t)0);
}

cudaError_t launch_sort_targets(const TargetBufs &b, long long n, int groups, const BBox *bb,
                                cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)((n + 255) / 256);
  size_t bytes = b.sort_bytes;
  cudaError_t e;
  if (groups == 1) {
    unsigned *k0 = reinterpret_cast<unsigned *>(b.keys), *k1 = k0 + n;
    launch_after(bs_target_keys<unsigned>, grid, 256, 0, s, b.tp_raw, b.tgroup, n, bb, k0, b.vals);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    e = cub::DeviceRadixSort::SortPairs(b.sort_tmp, bytes, (const unsigned *)k0, k1,
                                        (const int *)b.vals, b.perm, (int)n, 0, 31, s);
  } else {
    unsigned long long *k0 = b.keys, *k1 = k0 + n;
    launch_after(bs_target_keys<unsigned long long>, grid, 256, 0, s, b.tp_raw, b.tgroup, n, bb,
                 k0, b.vals);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    e = cub::DeviceRadixSort::SortPairs(b.sort_tmp, bytes, (const unsigned long long *)k0, k1,
                                        (const int *)b.vals, b.perm, (int)n, 0,
                                        31 + group_bits(groups), s);
  }
  return e != cudaSuccess ? e : launch_gather_targets(b.tp_raw, b.perm, n, b.tp, s);
}

cudaError_t launch_target_keys(const double4 *tp, long long n, const BBox *bb, float *keys,
                               cudaStream_t s) {
  launch_after(bs_target_keys<float>, (unsigned)((n + 255) / 256), 256, 0, s, tp,
               (const int *)nullptr, n, bb, keys, (int *)nullptr);
  return cudaGetLastError();
}

cudaError_t launch_order_targets(long long n, const TargetBufs &b, const BBox *bb, cudaStream_t s) {
  return launch_order_targets(OneGroup{(int)n}, 1, n, n, b, bb, s);
}

cudaError_t launch_reduce(const Tile *tiles, int n_tiles, const Group *groups, const double *part,
                          const int *perm, int tile_cap, unsigned *ctr, cudaStream_t s,
                          const Item *items, const GroupLive *live) {
  if (n_tiles <= 0) return cudaSuccess;
  if (live && !items) return cudaErrorInvalidValue;
  const dim3 grid((unsigned)n_tiles, (unsigned)(tile_cap + 31) / 32);
  launch_after(bs_reduce, grid, 32 * kReduceWarps, 0, s, tiles, groups, part, perm, tile_cap,
               items, live, ctr);
  return cudaGetLastError();
}

cudaError_t launch_length(const double *F1, const double *F2, long long d0, long long nf, double *L,
                          cudaStream_t s) {
  if (nf <= 0) return cudaSuccess;
  const int bs = 256;
  bs_length<<<(unsigned)((nf + bs - 1) / bs), bs, 0, s>>>(F1, F2, d0, nf, L);
  return cudaGetLastError();
}

unsigned long long default_wait_limit_ns() { return kDefaultWaitNs; }

cudaError_t launch_ffma_peak(float *out, int blocks, int iters, cudaStream_t s) {
  bs_ffma_peak<<<blocks, 256, 0, s>>>(out, iters, 0.999999f, 1e-7f);
  return cudaGetLastError();
}

cudaError_t launch_roots_selftest(const double *x, long long n, double *y, cudaStream_t s) {
  bs_roots_selftest<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(x, n, y);
  return cudaGetLastError();
}

cudaError_t launch_wait_selftest(unsigned *err, unsigned long long limit_ns, cudaStream_t s) {
  bs_wait_selftest<<<1, 32, 0, s>>>(err, limit_ns);
  return cudaGetLastError();
}

}  // namespace winds
