// kj_kernels.cu -- device kernels of the Kutta-Joukowski fixed point
// (core/KuttaJoukowski.m:42-49 and kj(), :173-298) for every case of a batch.
//   kj_targets   lifting-line points of step s -> direct-sum targets (:216-219)
//   kj_solve     the fixed point: every iteration of every case in one launch,
//                per station the blade-frame transform (:241-246), aoa (:258),
//                interp1 of the airfoil tables (:262-269), Γ = ½|V|c Cl (:277),
//                the relaxed update (:281) and the relative residual in FP64
//                (:290); a case stops when max |residual| <= tol (:45)
//   kj_finish    the batch's iteration count and the last induced velocities
//   kj_features, kj_apply_guess   inputs and result of the bound-circulation
//                MLP that replaces the previous-step start value (WInDS.m:131)
//   kj_loads     rotor thrust, torque and power (postproc/perform.m:18-62)
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "bs_device.cuh"
#include "bs_launch.h"
#include "kj_launch.h"
#include "wake_types.h"

namespace winds {

// Also the state an iteration starts from: none done, none converged.
__global__ void kj_targets(const WakeCase *cases, const KJCase *kc, const int *step,
                           const double *ll, double4 *tp, BBox *bb, int *iters, int *converged,
                           int *diverged, int *it_max) {
  after_previous();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    iters[blockIdx.y] = converged[blockIdx.y] = diverged[blockIdx.y] = 0;
    if (blockIdx.y == 0) *it_max = 0;
  }
  const WakeCase c = cases[blockIdx.y];
  const KJCase k = kc[blockIdx.y];
  const int ns = c.nst - 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  if (t < ns * c.nb) {
    const int i = t % ns, b = t / ns;
    const int s = *step;
    const double *p = ll + k.frame_off + i + (long long)ns * (3 * (s + (long long)c.nsteps * b));
    tp[k.t_off + t] = make_double4(p[0], p[ns], p[2 * ns], 0.0);
    for (int a = 0; a < 3; ++a) lo[a] = hi[a] = (float)p[a * ns];
  }
  bbox_accumulate(lo, hi, bb->tmin, bb->tmax);
}

// MATLAB interp1(x, y, xi) of two tables: linear, NaN outside [x(1), x(end)].
// lo: the interval of the last call, where the search starts (from one iteration to
// the next it seldom changes), and of this one.
__device__ void interp1(const double *x, const double *y, const double *z, int n, double xi,
                        double &yi, double &zi, int &last) {
  if (!(xi >= __ldg(x) && xi <= __ldg(x + n - 1))) {
    yi = zi = NAN;
    return;
  }
  int lo = last, hi = lo + 1;
  if (hi >= n || !(__ldg(x + lo) <= xi && xi < __ldg(x + hi))) {
    lo = 0, hi = n - 1;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(x + mid) <= xi) lo = mid; else hi = mid;
    }
    last = lo;
  }
  const double t = (xi - __ldg(x + lo)) / (__ldg(x + hi) - __ldg(x + lo));
  yi = __ldg(y + lo) + t * (__ldg(y + hi) - __ldg(y + lo));
  zi = __ldg(z + lo) + t * (__ldg(z + hi) - __ldg(z + lo));
}

// ---------------------------------------------------------------- kj_solve
// The iteration's Biot-Savart calls (KuttaJoukowski.m:216,218) differ from one
// iteration to the next only in the circulation of the filaments that follow
// the bound iterate -- shed columns 0 and 1 and trailing column 0, nb (2 ns +
// nst) "own" filaments -- and the velocity is linear in it. So the direct sum
// over all other filaments runs once per step (u_fix), and an iteration adds
// the own filaments' influence: a matrix of unit-circulation terms in FP64,
// formed once, times their circulation. Before, each iteration was six
// launches over every filament: 89 us for one rotor of 17 x 60 (23 us of it
// the sum), 30 iterations of it most of the step.
//
// A cluster of kCluster CTAs runs a case. Each CTA owns a slice of the
// lifting-line points: it forms their rows of the matrix in its shared memory
// (16 points x 363 filaments x 24 B on 41 nodes; beyond the limit the rows go to
// the global scratch, and with no scratch each term is formed again in each
// iteration), and every iteration a warp per point sums its row, updates its
// station and sends the new circulation to all CTAs of the cluster, each of which
// then forms all own circulations by itself. The values travel as asynchronous
// stores that complete on an mbarrier of the receiver: with a cluster barrier
// instead, 4300 of an iteration's 10000 cycles went into it. Latency bounds the
// rest: the row sums, the station update and the stores' way are one chain of some
// 5000 cycles (99 us for 30 iterations on 17 nodes; 124 with the span sums as a
// chain, a search of the whole table and a butterfly for the residual). Every
// loop ends after maxiter iterations, every wait within the time limit.
namespace cg = cooperative_groups;
constexpr int kCluster = 8;
constexpr int kSolveThreads = 512;
constexpr int kSolveWarps = kSolveThreads / 32;

// Endpoints, squared core and index of own filament f of case c: shed columns 0
// and 1 of each blade (b, j, i), then trailing column 0 (b, i).
struct OwnFilament {
  double4 A, B;
};
__device__ __forceinline__ OwnFilament own_filament(const WakeCase &c, const double *dom,
                                                    const double *rc_s, const double *rc_t, int f) {
  const int ns = c.nst - 1, n_shed = c.nb * 2 * ns;
  int i, j, b, j1, j2, i2;
  double rc;
  if (f < n_shed) {
    b = f / (2 * ns);
    const int r = f - b * 2 * ns;
    j = r / ns;
    i = r - j * ns;
    j1 = j2 = j;
    i2 = i + 1;
    rc = rc_s[c.shed_off + i + (long long)ns * (j + (long long)c.na * b)];
  } else {
    const int u = f - n_shed;
    b = u / c.nst;
    i = i2 = u - b * c.nst;
    j1 = 1, j2 = 0;
    rc = rc_t[c.trail_off + i + (long long)c.nst * ((long long)(c.na - 1) * b)];
  }
  const double *p1 = dom + c.node_off * 3 + i + (long long)c.nst * 3 * (j1 + (long long)c.na * b);
  const double *p2 = dom + c.node_off * 3 + i2 + (long long)c.nst * 3 * (j2 + (long long)c.na * b);
  OwnFilament o;
  o.A = make_double4(p1[0], p1[c.nst], p1[2 * c.nst], 1.0);
  o.B = make_double4(p2[0], p2[c.nst], p2[2 * c.nst], rc);
  return o;
}

// What a station's update reads besides the velocity, gathered once per step:
// the frame (9), vblade (3), |vblade| chord / 2 and the fixed velocity (3); and
// what its last update gave: the velocity (3), cl, cd and aoa, kept here until
// the end (a store to global memory would hold up every cluster barrier).
constexpr int kStation = 24;
__device__ __forceinline__ void load_station(const KJSolveArgs &a, const WakeCase &c,
                                             const KJCase &k, int s, int t, double *st) {
  const int ns = c.nst - 1, b = t / ns, i = t - b * ns;
  const long long fo = k.frame_off + i + (long long)ns * (3 * (s + (long long)c.nsteps * b));
  const double *fr[3] = {a.bxn, a.byn, a.bzn};
  const double *fix = a.u_fix + 3 * k.t_off + i + (long long)ns * 3 * b;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
#pragma unroll
    for (int r = 0; r < 3; ++r) st[3 * q + r] = fr[q][fo + r * ns];
    st[9 + q] = a.vblade[fo + q * ns];
    st[13 + q] = fix[q * ns];
  }
  st[12] = 0.5 * sqrt(st[9] * st[9] + st[10] * st[10] + st[11] * st[11]) *
           a.chord[k.station_off + i];
  int *table = reinterpret_cast<int *>(st + 22);
  const int fo2 = k.foil_base + a.foil[k.station_off + i];
  table[0] = a.foil_off[fo2], table[1] = a.foil_off[fo2 + 1], table[2] = 0;
}

// A station's update with induced velocity u; returns the updated circulation,
// the residual's bits in *res (0, and the circulation unchanged, where Cl is
// NaN).
__device__ __forceinline__ double station_update(const KJSolveArgs &a, double *st, int ci,
                                                 const double u[3], double bound,
                                                 unsigned long long *res) {
  double rot[3];
#pragma unroll
  for (int q = 0; q < 3; ++q)
    rot[q] = st[3 * q] * u[0] + st[3 * q + 1] * u[1] + st[3 * q + 2] * u[2];
  const double tu = st[9] + rot[0], tv = st[10] + rot[1];
  const double aoa = atan2(-tv, tu) * (180.0 / kPi);
  double cl, cd;
  int *table = reinterpret_cast<int *>(st + 22);
  const int o0 = table[0];
  interp1(a.aoa_t + o0, a.cl_t + o0, a.cd_t + o0, table[1] - o0, aoa, cl, cd, table[2]);
  st[16] = u[0], st[17] = u[1], st[18] = u[2];
  st[19] = cl, st[20] = cd, st[21] = aoa;
  *res = 0ull;
  if (isnan(cl)) {
    atomicOr(&a.diverged[ci], 1);
    return bound;
  }
  const double gamma = st[12] * cl;
  const double dg = gamma - bound;
  *res = (unsigned long long)__double_as_longlong(fabs(dg / (fabs(gamma) + 1.0)));
  return bound + a.relax * dg;
}

// Address in CTA `rank` of the cluster of the shared-memory address p is here.
__device__ __forceinline__ uint32_t cluster_address(const void *p, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
// (g, r) to 16 bytes of another CTA's shared memory, completing on its mbarrier.
__device__ __forceinline__ void send_pair(uint32_t dst, uint32_t bar, double g,
                                          unsigned long long r) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(
          dst),
      "l"((unsigned long long)__double_as_longlong(g)), "l"(r), "r"(bar)
      : "memory");
}

__global__ void __launch_bounds__(kSolveThreads) kj_solve(const KJSolveArgs a) {
  after_previous();
  extern __shared__ __align__(16) double kj_smem[];
  __shared__ uint64_t arrived[2];
  cg::cluster_group cl = cg::this_cluster();
  const int ci = blockIdx.x / kCluster, rank = blockIdx.x % kCluster;
  const WakeCase c = a.cases[ci];
  const KJCase k = a.kc[ci];
  const int s = *a.step;
  const int ns = c.nst - 1, nt = ns * c.nb, n_shed = c.nb * 2 * ns, own = n_shed + c.nb * c.nst;
  const int per = (nt + kCluster - 1) / kCluster;
  const int t0 = rank * per;
  const int cnt = max(0, min(per, nt - t0));
  // CTAs of the exchange: those that own points (42 points leave the last none, as
  // fewer than 8 leave several). Nobody would wait for another, so a buffer it still
  // reads would be filled again; it goes on to the end. With the vectors in memory
  // cluster barriers keep all CTAs in step.
  const int parts = a.vec_smem ? (nt + per - 1) / per : kCluster;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int tt = tid; tt < cnt; tt += kSolveThreads)  // the start value, kept for the caller
    a.guess[c.bound_off + t0 + tt] = a.bound[c.bound_off + t0 + tt];
  if (s < c.kj_from) return;  // the start-up's first step has no iteration
  // shared or (vectors too long for it) global working vectors: the bound
  // iterate and the residual (its bits) of every point, twice; the own circulations; the
  // part of shed column 1 that stays; this CTA's stations (load_station)
  double *vec = a.vec_smem ? kj_smem : a.vec_scratch + ((long long)ci * kCluster + rank) * a.vec_stride;
  double2 *sB[2] = {reinterpret_cast<double2 *>(vec), reinterpret_cast<double2 *>(vec + 2 * nt)};
  double *sG = vec + 4 * nt, *sC = sG + own, *sS = sC + nt;
  double *mat = a.mat_smem      ? kj_smem + (a.vec_smem ? a.vec_stride : 0)
                : a.mat_scratch ? a.mat_scratch + ((long long)ci * kCluster + rank) * a.mat_stride
                                : nullptr;
  RefParams rp;
  rp.model = a.model;
  rp.d = a.d;
  rp.n = a.n;
  rp.co = a.co;
  const auto term = [&](int tt, int f, double u[3]) {
    const double4 p = a.tp[k.t_off + t0 + tt];
    const OwnFilament o = own_filament(c, a.dom, a.rc_s, a.rc_t, f);
    u[0] = u[1] = u[2] = 0.0;
    ref_pair(o.A, o.B, p.x, p.y, p.z, rp, u[0], u[1], u[2]);
  };
  if (mat)
    for (int idx = tid; idx < cnt * own; idx += kSolveThreads) {
      const int tt = idx / own, f = idx - tt * own;
      double u[3];
      term(tt, f, u);
#pragma unroll
      for (int q = 0; q < 3; ++q) mat[(long long)(3 * tt + q) * own + f] = u[q];
    }
  for (int t = tid; t < nt; t += kSolveThreads) sB[0][t].x = a.bound[c.bound_off + t];
  if (tid == 0) {
    mbar_init(&arrived[0], 1);
    mbar_init(&arrived[1], 1);
    fence_mbar_init();
  }
  for (int tt = tid; tt < cnt; tt += kSolveThreads)
    load_station(a, c, k, s, t0 + tt, sS + kStation * tt);
  // shed(:, 1) = C_1 - C_0 (WInDS.m:139-140): C_1, of the previous step's
  // trailing column 0, stays; summed as wake_bookkeep does
  const int m = live_cols(c, s) - 1;
  for (int b = tid; b < c.nb; b += kSolveThreads) {
    double cum = 0.0;
    const double *tp = a.trail_prev + c.trail_off + (long long)c.nst * ((long long)(c.na - 1) * b);
    for (int i = 0; i < ns; ++i) {
      if (m > 1) cum += tp[i];
      sC[i + ns * b] = cum;
    }
  }
  cl.sync();
  // the own circulations of iterate B; a non-finite one adds nothing, as its
  // terms are zeroed in the direct sum (BiotSavart.m:111)
  const auto circulation = [&](const double2 *B) {
    const auto put = [&](int f, double g) { sG[f] = isfinite(g) ? g : 0.0; };
    bool bad = false;
    for (int t = tid; t < c.nb * c.nst; t += kSolveThreads) {
      const int b = t / c.nst, i = t - b * c.nst;
      const double hi = i < ns ? B[i + ns * b].x : 0.0, lo = i > 0 ? B[i - 1 + ns * b].x : 0.0;
      bad = bad || !isfinite(hi);
      put(n_shed + t, hi - lo);
      // shed column 1: C_1 - C_0, where C_0, a running sum of differences from the
      // first station on, is hi itself (formed as a sum it took 1200 of 6700 cycles)
      if (i < ns) put(2 * ns * b + i, hi), put(2 * ns * b + ns + i, sC[i + ns * b] - hi);
    }
    if (!__syncthreads_or(bad)) return;
    // unless one is not finite, which the sum passes on to the stations after it
    for (int b = tid; b < c.nb; b += kSolveThreads) {
      double cum = 0.0;
      for (int i = 0; i < ns; ++i) {
        cum += B[i + ns * b].x - (i > 0 ? B[i - 1 + ns * b].x : 0.0);
        put(2 * ns * b + ns + i, sC[i + ns * b] - cum);
      }
    }
    __syncthreads();
  };
  // velocity at point tt of this CTA, in every lane of the warp
  const auto velocity = [&](int tt, double u[3]) {
    double v[3] = {0.0, 0.0, 0.0};
    if (mat) {
      const double *r = mat + (long long)3 * tt * own;
#pragma unroll 4
      for (int f = lane; f < own; f += 32) {
        const double g = sG[f];
        v[0] = fma(r[f], g, v[0]);
        v[1] = fma(r[own + f], g, v[1]);
        v[2] = fma(r[2 * own + f], g, v[2]);
      }
    } else {
      for (int f = lane; f < own; f += 32) {
        double w[3];
        term(tt, f, w);
        const double g = sG[f];
#pragma unroll
        for (int q = 0; q < 3; ++q) v[q] = fma(w[q], g, v[q]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < 3; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
#pragma unroll
    for (int q = 0; q < 3; ++q) u[q] = sS[kStation * tt + 13 + q] + v[q];
  };
  int it = 0;
  bool done = false;
  double res = 0.0;
  while (rank < parts && it < a.maxiter && !done) {
    const int cur = it & 1, nxt = cur ^ 1;
    if (a.vec_smem && tid == 0) mbar_arrive_expect_tx(&arrived[nxt], 16u * (unsigned)nt);
    circulation(sB[cur]);
    for (int tt = warp; tt < cnt; tt += kSolveWarps) {
      double u[3];
      velocity(tt, u);
      const int t = t0 + tt, b = t / ns, i = t - b * ns;
      double g = 0.0;
      unsigned long long r = 0ull;
      if (lane == 0) {
        g = station_update(a, sS + kStation * tt, ci, u, sB[cur][t].x, &r);
      }
      g = __shfl_sync(0xffffffffu, g, 0);
      r = __shfl_sync(0xffffffffu, r, 0);
      if (lane < parts) {
        // a buffer is written again only after every CTA of the exchange sent what
        // it formed from it, two iterations on
        if (a.vec_smem)
          send_pair(cluster_address(sB[nxt] + t, lane), cluster_address(&arrived[nxt], lane), g, r);
        else
          reinterpret_cast<double2 *>(reinterpret_cast<double *>(sB[nxt]) +
                                      ((long long)lane - rank) * a.vec_stride)[t] =
              make_double2(g, __longlong_as_double((long long)r));
      }
    }
    if (a.vec_smem) {
      // iteration it fills buffer nxt for the (it / 2)-th time
      const bool ok = mbar_wait_bounded(&arrived[nxt], (unsigned)(it >> 1) & 1u, a.err, a.wait_limit_ns);
      if (!__syncthreads_and(ok)) break;
    } else {
      cl.sync();
    }
    unsigned long long r = 0ull;  // largest residual: the bits of non-negative doubles order them
    for (int t = lane; t < nt; t += 32) r = max(r, (unsigned long long)__double_as_longlong(sB[nxt][t].y));
    const unsigned top = __reduce_max_sync(0xffffffffu, (unsigned)(r >> 32));
    const unsigned low = __reduce_max_sync(0xffffffffu, (unsigned)(r >> 32) == top ? (unsigned)r : 0u);
    r = (unsigned long long)top << 32 | low;
    res = __longlong_as_double((long long)r);
    done = res <= a.tol;
    ++it;
  }
  for (int tt = tid; tt < cnt; tt += kSolveThreads) {
    const int t = t0 + tt, b = t / ns, i = t - b * ns;
    const double *st = sS + kStation * tt;
    double *o = a.uindb + 3 * k.t_off + i + (long long)ns * 3 * b;  // [ns,3,nb] of this case
#pragma unroll
    for (int q = 0; q < 3; ++q) o[q * ns] = st[16 + q];
    a.cl_out[c.bound_off + t] = st[19];
    a.cd_out[c.bound_off + t] = st[20];
    a.aoa_out[c.bound_off + t] = st[21];
    a.bound[c.bound_off + t] = sB[it & 1][t].x;
  }
  if (done) {
    // the velocities of the converged circulation, for kj_finish
    circulation(sB[it & 1]);
    for (int tt = warp; tt < cnt; tt += kSolveWarps) {
      double u[3];
      velocity(tt, u);
      const int t = t0 + tt, b = t / ns, i = t - b * ns;
      double *o = a.uindb_conv + 3 * k.t_off + i + (long long)ns * 3 * b;
      if (lane == 0)
#pragma unroll
        for (int q = 0; q < 3; ++q) o[q * ns] = u[q];
    }
  }
  if (rank == 0 && tid == 0) {
    a.iters[ci] = it;
    a.converged[ci] = done;
    a.res_last[ci] = res;
    atomicMax(a.it_max, it);
  }
  cl.sync();  // no CTA leaves while another may still read or write its shared memory
}

// A case that converged before the batch's last iteration ends with the
// induced velocity of its converged circulation, as if it had been evaluated
// with the others to the end.
__global__ void kj_finish(const WakeCase *cases, const KJCase *kc, const int *iters,
                          const int *converged, const int *it_max, const double *uindb_conv,
                          double *uindb) {
  after_previous();
  const int ci = blockIdx.y;
  const int n = 3 * (cases[ci].nst - 1) * cases[ci].nb;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n || !converged[ci] || iters[ci] >= *it_max) return;
  uindb[3 * kc[ci].t_off + t] = uindb_conv[3 * kc[ci].t_off + t];
}

// The inflow features are the station's total inflow in the blade frame at
// this step with the induced velocity of the previous step's last iteration
// (uindb, zero before the first step): vblade + [bxn; byn; bzn] uindb, the
// velocity the first iteration of kj() would see (core/KuttaJoukowski.m:241-249).
// The history: bound (the last converged value), bound_last and bound_last2
// (the two before it; equal to bound before there were any), which move one step
// on here for the next step's change features.
__global__ void kj_features(const WakeCase *cases, const KJCase *kc, const int *step,
                            const double *bound, double *bound_last, double *bound_last2,
                            const double *vblade, const double *bxn,
                            const double *byn, const double *bzn, const double *uindb,
                            const double *st_r, const double *st_c, const double *st_tw,
                            const double *azim, float *x) {
  after_previous();
  const WakeCase c = cases[blockIdx.y];
  const KJCase k = kc[blockIdx.y];
  const int ns = c.nst - 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ns * c.nb) return;
  const int i = t % ns, b = t / ns;
  const int s = *step;
  const long long fo = k.frame_off + i + (long long)ns * (3 * (s + (long long)c.nsteps * b));
  const long long st = k.station_off + i;
  const double az = azim[k.az_off + s + (long long)c.nsteps * b];
  float *f = x + (k.t_off + t) * kKJFeatures;
  f[0] = (float)st_r[st];
  f[1] = (float)st_c[st];
  f[2] = (float)st_tw[st];
  f[3] = (float)sin(az);
  f[4] = (float)cos(az);
  const double *u = uindb + 3 * k.t_off + i + (long long)ns * 3 * b;
  const double *fr[3] = {bxn, byn, bzn};
  for (int a = 0; a < 3; ++a)
    f[5 + a] = (float)(vblade[fo + a * ns] +
                       (fr[a][fo] * u[0] + fr[a][fo + ns] * u[ns] + fr[a][fo + 2 * ns] * u[2 * ns]));
  const long long q = c.bound_off + i + (long long)ns * b;
  const double g0 = bound[q], g1 = bound_last[q], g2 = bound_last2[q];
  f[8] = (float)g0;
  f[9] = (float)(g0 - g1);
  f[10] = (float)(g1 - g2);
  bound_last[q] = g0;
  bound_last2[q] = g1;
}

// bound = base + out_scale * y, base Gamma_prev or, with *base != 0, its
// extrapolation Gamma_prev + dGamma_prev (feature 9 of the row). Two kinds of
// station keep Gamma_prev: those whose airfoil table has no lift (st_lift 0:
// Cl = 0 at every AoA, e.g. the cylinder root sections; their fixed point is
// Gamma = 0, the previous step already sits there, and the relaxed iteration
// damps any start error there by only 1 - relax per iteration), and those
// whose last converged AoA (aoa_prev) lies outside their table's stall bounds
// st_stall (the AoA of its lowest and highest Cl) less kStallMargin degrees:
// past stall a station can have more than one fixed point, and the previous
// step's value is the start that keeps the branch it is on.
// Nothing before the step the iteration starts at (WakeCase::kj_from).
constexpr double kStallMargin = 2.0;  // degrees
__global__ void kj_apply_guess(const WakeCase *cases, const KJCase *kc, const int *step,
                               const int *st_lift, const double2 *st_stall,
                               const double *aoa_prev, const float *y, const float *out_scale,
                               const float *feat, const float *base, double *bound) {
  after_previous();
  const WakeCase c = cases[blockIdx.y];
  const KJCase k = kc[blockIdx.y];
  const int ns = c.nst - 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ns * c.nb || *step < c.kj_from) return;
  const int i = t % ns, b = t / ns;
  if (!st_lift[k.station_off + i]) return;
  const double2 sb = st_stall[k.station_off + i];
  const double ap = aoa_prev[c.bound_off + i + (long long)ns * b];
  if (!(ap > sb.x + kStallMargin && ap < sb.y - kStallMargin)) return;
  double g = bound[c.bound_off + i + (long long)ns * b];
  if (*base != 0.f) g += (double)feat[(k.t_off + t) * kKJFeatures + 9];
  bound[c.bound_off + i + (long long)ns * b] = g + (double)*out_scale * (double)y[k.t_off + t];
}

// Spanwise loads of one station (postproc/perform.m:20-55): the blade-frame
// velocity to the rotor frame, velX = -Rz(theta - 90 deg) vblade with theta =
// twist + pitch (DCMRot with the 'zzz' sequence [-90, twist, pitch]); inflow
// angle phi = aoa - theta; a/a' = TSR / tan(phi); a and a'; normal and
// tangential coefficients; dT, dQ, dP.
__global__ void kj_dloads(const WakeCase *cases, const KJCase *kc, const int *step,
                          const double *vblade, const double *cl, const double *cd,
                          const double *aoa, const double *st_tw, const double *chord,
                          const double *st_rr, const double *st_dr, const double *rpm,
                          const double *pitch, double *dl) {
  after_previous();
  const WakeCase c = cases[blockIdx.y];
  const KJCase k = kc[blockIdx.y];
  const int ns = c.nst - 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ns * c.nb) return;
  const int i = t % ns, b = t / ns;
  const int s = *step;
  const long long fo = k.frame_off + i + (long long)ns * (3 * (s + (long long)c.nsteps * b));
  const long long st = k.station_off + i;
  const long long q = c.bound_off + i + (long long)ns * b;
  double th = st_tw[st] * (180.0 / kPi);  // deg
  if (k.has_pitch) th += pitch[k.az_off + s + (long long)c.nsteps * b];
  const double rot = (th - 90.0) * (kPi / 180.0);
  const double cr = cos(rot), sr = sin(rot);
  const double u0 = vblade[fo], u1 = vblade[fo + ns];
  const double v1 = -(cr * u0 - sr * u1);
  const double v2 = -(sr * u0 + cr * u1);
  const double tsr = v2 / v1;
  const double phi = aoa[q] - th;
  const double pr = phi * (kPi / 180.0);
  const double tp = tan(pr);
  const double aap = tsr / tp;
  const double a = aap * (v1 - tp * v2) / (aap * v1 + tp * v2);
  const double ap = a / aap;
  const double cz = cl[q] * cos(pr) + cd[q] * sin(pr);
  const double cx = cl[q] * sin(pr) - cd[q] * cos(pr);
  const double w1 = v1 * (1.0 - a), w2 = v2 * (1.0 + ap);
  const double w = w1 * w1 + w2 * w2;
  const double dT = 0.5 * k.rho * chord[st] * cz * w * st_dr[st];
  const double dQ = 0.5 * k.rho * chord[st] * cx * w * st_rr[st] * st_dr[st];
  double *o = dl + 3 * (k.t_off + t);
  o[0] = dT;
  o[1] = dQ;
  o[2] = (kPi / 30.0) * rpm[k.rpm_off + s] * dQ;
}

// Rotor totals, summed over stations and then blades as sum(sum(dT,1),4).
__global__ void kj_sum_loads(const WakeCase *cases, const KJCase *kc, int ncases,
                             const double *dl, double *out) {
  after_previous();
  const int ci = blockIdx.x * blockDim.x + threadIdx.x;
  if (ci >= ncases) return;
  const WakeCase c = cases[ci];
  const KJCase k = kc[ci];
  const int ns = c.nst - 1;
  double tot[3] = {0.0, 0.0, 0.0};
  for (int b = 0; b < c.nb; ++b) {
    double sb[3] = {0.0, 0.0, 0.0};
    for (int i = 0; i < ns; ++i)
      for (int a = 0; a < 3; ++a) sb[a] += dl[3 * (k.t_off + i + (long long)ns * b) + a];
    for (int a = 0; a < 3; ++a) tot[a] += sb[a];
  }
  for (int a = 0; a < 3; ++a) out[3 * ci + a] = tot[a];
}

cudaError_t launch_kj_targets(const WakeCase *cases, const KJCase *kc, int ncases, int max_st,
                              const int *step, const double *ll, double4 *tp, BBox *bb, int *iters,
                              int *converged, int *diverged, int *it_max, cudaStream_t s) {
  launch_after(kj_targets, dim3((max_st + 127) / 128, ncases), 128, 0, s, cases, kc, step, ll, tp,
               bb, iters, converged, diverged, it_max);
  return cudaGetLastError();
}

// Doubles of a CTA's working vectors and matrix rows for a case of ns stations
// and nb blades.
long long kj_vec_doubles(int ns, int nb) {
  const long long n = 5LL * ns * nb + (long long)nb * (3 * ns + 1) +
                      (long long)kStation * ((ns * nb + kCluster - 1) / kCluster);
  return (n + 1) / 2 * 2;  // 16-byte strides
}
long long kj_mat_doubles(int ns, int nb) {
  return (long long)(ns * nb + kCluster - 1) / kCluster * 3 * nb * (3 * ns + 1);
}
int kj_cluster() { return kCluster; }

cudaError_t launch_kj_solve(const KJSolveArgs &a, int ncases, cudaStream_t s) {
  const size_t smem = (size_t)((a.vec_smem ? a.vec_stride : 0) + (a.mat_smem ? a.mat_stride : 0)) *
                      sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(kj_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kKJSmemBytes);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ncases * kCluster);
  cfg.blockDim = dim3(kSolveThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kCluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kj_solve, a);
}

cudaError_t launch_kj_finish(const WakeCase *cases, const KJCase *kc, int ncases, int max_st,
                             const int *iters, const int *converged, const int *it_max,
                             const double *uindb_conv, double *uindb, cudaStream_t s) {
  launch_after(kj_finish, dim3((3 * max_st + 127) / 128, ncases), 128, 0, s, cases, kc, iters,
               converged, it_max, uindb_conv, uindb);
  return cudaGetLastError();
}

cudaError_t launch_kj_features(const WakeCase *cases, const KJCase *kc, int ncases, int max_st,
                               const int *step, const double *bound, double *bound_last,
                               double *bound_last2, const double *vblade,
                               const double *bxn, const double *byn, const double *bzn,
                               const double *uindb, const double *st_r,
                               const double *st_c, const double *st_tw, const double *azim,
                               float *x, cudaStream_t s) {
  launch_after(kj_features, dim3((max_st + 127) / 128, ncases), 128, 0, s, cases, kc, step, bound,
               bound_last, bound_last2, vblade, bxn, byn, bzn, uindb, st_r, st_c, st_tw, azim, x);
  return cudaGetLastError();
}

cudaError_t launch_kj_apply_guess(const WakeCase *cases, const KJCase *kc, int ncases, int max_st,
                                  const int *step, const int *st_lift, const double2 *st_stall,
                                  const double *aoa_prev, const float *y, const float *out_scale,
                                  const float *feat, const float *base, double *bound,
                                  cudaStream_t s) {
  launch_after(kj_apply_guess, dim3((max_st + 127) / 128, ncases), 128, 0, s, cases, kc, step,
               st_lift, st_stall, aoa_prev, y, out_scale, feat, base, bound);
  return cudaGetLastError();
}

cudaError_t launch_kj_loads(const WakeCase *cases, const KJCase *kc, int ncases, int max_st,
                            const int *step, const double *vblade, const double *cl,
                            const double *cd, const double *aoa, const double *st_tw,
                            const double *chord, const double *st_rr, const double *st_dr,
                            const double *rpm, const double *pitch, double *dl, double *out,
                            cudaStream_t s) {
  launch_after(kj_dloads, dim3((max_st + 127) / 128, ncases), 128, 0, s, cases, kc, step, vblade,
               cl, cd, aoa, st_tw, chord, st_rr, st_dr, rpm, pitch, dl);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  launch_after(kj_sum_loads, (ncases + 127) / 128, 128, 0, s, cases, kc, ncases, dl, out);
  return cudaGetLastError();
}

}  // namespace winds
