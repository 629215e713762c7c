// Mean profiles (meanprofiles.F90), the mean-profile subsidence tendencies (forcing.F90) the
// damping and forcing components read, and the profile_diagnostics sums
// (profile_diagnostics.F90).
//
// MONC's mean_profiles runs in the solver group, after stepfields: olzubar, olzvbar, olzthbar and
// olzqbar are the horizontal means of the stepped fields before the pressure correction.  In the
// fused step those are zu_n, zv_n and the new theta and q; the next step's damping and forcing
// read them.  Each level of each field is summed in a fixed order (deterministic), in FP64 whatever
// the field precision, and multiplied by rnhpts = 1 / real(nx ny) as MONC does.
#include "dycore.h"
#include "dycore_device.cuh"
#include "level_sums.cuh"

namespace mgpu {

// Level sums over a cluster of blocks (level_sums.cuh); all profiles of a step in one launch.
constexpr int PT = 256;

// sums v[q] of the block's threads (in place in thread 0): warp shuffles, then the warps in order
template <int NV>
__device__ __forceinline__ void block_sums(double (&v)[NV], double (*sh)[PT / 32]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q)
    for (int h = 16; h; h >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], h);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) sh[q][w] = v[q];
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double a = 0.0;
      for (int x = 0; x < PT / 32; ++x) a += sh[q][x];
      sh[q][0] = a;
    }
}

// How many blocks (1, 2, 4 or 8) share a level of `points` points, for `sums` level sums in all: the number
// with the least waves x (a block's points + `fixed`), fixed standing for what a block costs besides its
// points and 5% a doubling for the cluster.  FP64, a call with its wait, for 1, 2, 4, 8 blocks, [chosen]:
//   six means    64 x 64 x 1000 [47] 53 74 155, 256 x 128 x 60 32 [23] 25 26, 1024 x 1024 x 20 603 322 192 [156] us
//   diagnostics  64 x 64 x 1000 [93] 101 120 181, 256 x 128 x 60 95 70 [46] 58, 1024 x 1024 x 20 4663 2368 1173 [619]
// (always eight blocks lost on deep grids of small levels, one block on few or large levels).  `slots` are the
// blocks resident on the 148 SMs of a B200, a constant so that the order of the sums does not depend on the device.
constexpr int SPLIT_SMS = 148;
static int level_split(long long points, long long sums, int slots, double fixed) {
  int best = 1;
  double best_cost = 0.0, penalty = 1.0;
  for (int n = 1; n <= PSPLIT; n *= 2, penalty += 0.05) {
    const long long waves = (sums * n + slots - 1) / slots;
    const double cost = (double)waves * ((double)points / n + fixed) * penalty;
    if (n == 1 || cost < best_cost) { best = n; best_cost = cost; }
  }
  return best;
}
// kernel on `split` blocks a cluster for each of levels x rows sums
template <typename... P, typename... A>
static void launch_split(void (*kernel)(P...), int split, int levels, int rows, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = split;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(split, levels, rows);
  cfg.blockDim = dim3(PT, 1, 1);
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

// field q of a mean: c[q] + p[q], or a[q] p[q] + b[q] p2[q] when p2[q] is set (theta after
// stepfields' time smoothing); row q of the result starts at out[q]
constexpr int MAX_MEANS = 2 * (3 + MGPU_MAX_Q);
template <typename T>
struct MeanRows {
  const T* p[MAX_MEANS];
  const T* p2[MAX_MEANS];
  double a[MAX_MEANS], b[MAX_MEANS], c[MAX_MEANS];
  double* out[MAX_MEANS];
  int n;
};

// the level sums run over count points from row offset off of each plane (a slab's interior rows)
template <typename T>
__global__ void __launch_bounds__(PT)
    k_plane_means(const __grid_constant__ MeanRows<T> f, long long plane, long long off, long long count, double rnhpts) {
  const int k = blockIdx.y + 1, q = blockIdx.z, r = blockIdx.x, split = gridDim.x;
  const long long chunk = (count + split - 1) / split, t0 = r * chunk, t1 = min(count, t0 + chunk);
  const long long base = (long long)(k - 1) * plane + off;
  const T* __restrict__ p = f.p[q] + base;
  const T* __restrict__ p2 = f.p2[q] ? f.p2[q] + base : nullptr;
  const double a = f.a[q], b = f.b[q], c = f.c[q];
  double acc[1] = {0.0};
  if (p2) {
#pragma unroll 4
    for (long long t = t0 + threadIdx.x; t < t1; t += PT) acc[0] += a * (double)__ldg(p + t) + b * (double)__ldg(p2 + t);
  } else {
#pragma unroll 4
    for (long long t = t0 + threadIdx.x; t < t1; t += PT) acc[0] += c + (double)__ldg(p + t);
  }
  __shared__ double sh[1][PT / 32];
  block_sums<1>(acc, sh);
  double tot[1] = {sh[0][0]};
  if (split > 1) cluster_total<1>(sh, tot);
  if (r == 0 && threadIdx.x == 0) f.out[q][k] = tot[0] * rnhpts;
}

// rnhpts of meanprofiles.F90:44: the point count converted at default (single) precision; a
// slab (halo rows above and below) averages its interior rows, which the slabs' driver averages
// again across the slabs (all slabs hold the same number of rows)
static long long interior(const Scalars& s, int halo) { return (long long)s.nx * (s.ny - 2 * halo); }
static double rnhpts(const Scalars& s, int halo) { return 1.0 / (double)(float)interior(s, halo); }

// olzubar, olzvbar, olzthbar and olzqbar(n): the means of zu, zv, theta and the q fields
template <typename T>
static void add_olz(MeanRows<T>& f, const Scalars& s, const T* zu, const T* zv, const T* th, const T* const* q, double* olz) {
  const T* p[3] = {zu, zv, th};
  for (int n = 0; n < 3 + s.nq; ++n, ++f.n) {
    f.p[f.n] = n < 3 ? p[n] : q[n - 3];
    f.out[f.n] = olz + (long long)n * (s.nz + 2);
  }
}
// olubar, olvbar, olthbar and olqbar(n): the means of ugal + u, vgal + v, theta and each q field,
// the scalars time-smoothed (c1 f + c2 zf) where their z-fields are given
template <typename T>
static void add_olbar(MeanRows<T>& f, const Scalars& s, const T* u, const T* v, const T* th, const T* zth,
                      const T* const* q, const T* const* zq, double ugal, double vgal, double c1, double c2, double* olbar) {
  const int nq = q ? s.nq : 0;
  for (int n = 0; n < 3 + nq; ++n, ++f.n) {
    const int m = f.n;
    f.out[m] = olbar + (long long)n * (s.nz + 2);
    if (n < 2) {
      f.p[m] = n == 0 ? u : v;
      f.c[m] = n == 0 ? ugal : vgal;
    } else {
      f.p[m] = n == 2 ? th : q[n - 3];
      f.p2[m] = n == 2 ? zth : (zq ? zq[n - 3] : nullptr);
      f.a[m] = c1;
      f.b[m] = c2;
    }
  }
}
template <typename T>
static int launch_means(const MeanRows<T>& f, const Scalars& s, cudaStream_t st, int halo) {
  launch_split(k_plane_means<T>, level_split(interior(s, halo), (long long)s.nz * f.n, 8 * SPLIT_SMS, 16000.0), s.nz, f.n, st, f, s.plane,
               (long long)halo * s.nx, interior(s, halo), rnhpts(s, halo));
  return 1;
}

template <typename T>
int launch_mean_profiles(const Scalars& s, const MeanProfileFields<T>& m, double* olz, double* olbar, cudaStream_t st,
                         int halo) {
  MeanRows<T> f{};
  add_olz(f, s, m.zu, m.zv, m.zs, m.zqs, olz);
  add_olbar(f, s, m.u, m.v, m.th, m.zth, m.q, m.zq, m.ugal, m.vgal, m.c1, m.c2, olbar);
  return launch_means(f, s, st, halo);
}
template int launch_mean_profiles<float>(const Scalars&, const MeanProfileFields<float>&, double*, double*, cudaStream_t, int);
template int launch_mean_profiles<double>(const Scalars&, const MeanProfileFields<double>&, double*, double*, cudaStream_t, int);

// profile_diagnostics (profile_diagnostics.F90:311-636, PW flow and TVD scalars): a level's blocks sum
// the MGPU_PD_* quantities over the plane in FP64, in a fixed order.  Bound by its loads' latency: two points
// a thread are in flight at three blocks an SM (80 registers; one point 5% slower, four blocks with one point
// 20% faster where the levels alone fill the chip and 5% slower on large levels).
template <typename T>
__global__ void __launch_bounds__(PT, 3) k_profile_diagnostics(Scalars s, const T* __restrict__ u,
                                                             const T* __restrict__ v, const T* __restrict__ w,
                                                             const T* __restrict__ th, const T* __restrict__ qv,
                                                             const T* __restrict__ ql, const double* __restrict__ olbar,
                                                             int has_mean, int halo, double* __restrict__ out) {
  constexpr int NR = MGPU_PD_COUNT;
  const int k = blockIdx.y + 1, r0 = blockIdx.x, nz = s.nz, st = nz + 2;
  const Geo g{s.nx, s.ny, s.nz, s.plane};
  auto P = [&](int id, int kk) { return s.prof[id * st + kk]; };
  const bool moist = qv != nullptr;
  double acc[NR];
  for (int r = 0; r < NR; ++r) acc[r] = 0.0;
  const double ugal = s.ugal, vgal = s.vgal, thref = P(P_THREF, k);
  const double thbar = olbar[2 * st + k];
  const double umean = (k < nz && has_mean) ? 0.5 * (olbar[k] + olbar[k + 1]) : 0.0;
  const double vmean = (k < nz && has_mean) ? 0.5 * (olbar[st + k] + olbar[st + k + 1]) : 0.0;
  // (a level has fewer than 2^31 points; a thread's next point is PT points on, without a division)
  const unsigned nx = s.nx, count = nx * (unsigned)(s.ny - 2 * halo);
  const unsigned chunk = (count + gridDim.x - 1) / gridDim.x, t1 = min(count, (r0 + 1) * chunk);
  const unsigned t0 = r0 * chunk + threadIdx.x, dj = PT / nx, di = PT % nx;
  unsigned row = t0 / nx, ix = t0 - row * nx;
#pragma unroll 2
  for (unsigned t = t0; t < t1; t += PT) {
    const int j = halo + (int)row, i = (int)ix;
    row += dj;
    ix += di;
    if (ix >= nx) { ix -= nx; ++row; }
    const long long o = g.at(k, j, i);
    const double w0 = (double)w[o], th0 = (double)th[o];
    acc[MGPU_PD_U_WIND] += (double)u[o] + ugal;
    acc[MGPU_PD_V_WIND] += (double)v[o] + vgal;
    acc[MGPU_PD_WW] += w0 * w0;
    if (k >= 2) {
      acc[MGPU_PD_W_WIND] += w0;
      acc[MGPU_PD_WWW] += w0 * w0 * w0;
      acc[MGPU_PD_WWWW] += (w0 * w0) * (w0 * w0);
    }
    acc[MGPU_PD_THETA] += th0 + thref;
    const double dth = th0 - thbar;
    acc[MGPU_PD_TH2] += dth * dth;
    if (k < nz) {
      const long long o1 = o + s.plane;
      if (k >= 2) acc[MGPU_PD_WTHETA_CN] += w0 * (0.5 * (th0 + (double)th[o1]));
      double up = 0.25 * ((double)u[o] + (double)u[g.at(k, j, i - 1)] + (double)u[o1] + (double)u[g.at(k + 1, j, i - 1)]) + ugal;
      up = up - umean;
      acc[MGPU_PD_UW] += up * w0;
      double vp = 0.25 * ((double)v[o] + (double)v[g.at(k, j - 1, i)] + (double)v[o1] + (double)v[g.at(k + 1, j - 1, i)]) + vgal;
      vp = vp - vmean;
      acc[MGPU_PD_VW] += vp * w0;
    }
    if (moist) {
      const double q0 = (double)qv[o], l0 = (double)ql[o];
      acc[MGPU_PD_VAPOUR] += q0;
      acc[MGPU_PD_LIQUID] += l0;
      if (k >= 2 && k < nz) {
        acc[MGPU_PD_WQV_CN] += 0.5 * (q0 + (double)qv[o + s.plane]) * w0;
        acc[MGPU_PD_WQL_CN] += 0.5 * (l0 + (double)ql[o + s.plane]) * w0;
      }
      const double tk = (th0 + thref) * P(P_RPREFRCP, k), pmb = P(P_PREFN, k) / 100.;
      acc[MGPU_PD_RH] += q0 / qsaturation<double>(tk, pmb);
    }
  }
  __shared__ double sh[NR][PT / 32];
  block_sums<NR>(acc, sh);
  if (gridDim.x > 1) {
    double tot[NR];
    cluster_total<NR>(sh, tot);
    if (r0 == 0 && threadIdx.x == 0)
#pragma unroll
      for (int r = 0; r < NR; ++r) sh[r][0] = tot[r];
  }
  const int nrows = moist ? NR : MGPU_PD_VAPOUR;
  if (r0 == 0 && threadIdx.x == 0)
    for (int r = 0; r < nrows; ++r) out[(size_t)r * nz + k - 1] = sh[r][0];
}

template <typename T>
int launch_profile_diagnostics(const Scalars& s, const T* u, const T* v, const T* w, const T* th, const T* qv,
                               const T* ql, const double* olbar, bool has_mean, double* out, cudaStream_t st,
                               int halo) {
  launch_split(k_profile_diagnostics<T>, level_split(interior(s, halo), s.nz, 3 * SPLIT_SMS, 1000.0), s.nz, 1, st, s, u, v, w, th, qv, ql,
               olbar, has_mean ? 1 : 0, halo, out);
  return 1;
}
template int launch_profile_diagnostics<float>(const Scalars&, const float*, const float*, const float*, const float*,
                                               const float*, const float*, const double*, bool, double*, cudaStream_t,
                                               int);
template int launch_profile_diagnostics<double>(const Scalars&, const double*, const double*, const double*,
                                                const double*, const double*, const double*, const double*, bool,
                                                double*, cudaStream_t, int);

// subsidence tendencies of the mean profiles (forcing.F90:1052-1166 with the profiles olzubar,
// olzvbar, olzthbar + thref and olzqbar), levels 2..nz: rows usub, vsub, thsub, qsub(n)
__global__ void k_subsidence_tendencies(Scalars s, const double* __restrict__ olz, double* __restrict__ tend,
                                        int flow_theta, int q) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int nz = s.nz, st = nz + 2;
  if (k > nz) return;
  auto P = [&](int id, int kk) { return s.prof[id * st + kk]; };
  if (flow_theta) {
    for (int r = 0; r < 2; ++r) {
      const double* prof = olz + r * st;
      double sub;
      if (k < nz)
        sub = 2.0 * (P(P_WSUBS, k - 1) * P(P_TZC1, k) * (prof[k] - prof[k - 1]) +
                     P(P_WSUBS, k) * P(P_TZC2, k) * (prof[k + 1] - prof[k]));
      else
        sub = 2.0 * (P(P_WSUBS, k - 1) * P(P_TZC1, k) * (prof[k] - prof[k - 1]));
      tend[r * st + k] = sub;
    }
    const double* th = olz + 2 * st;
    const int ka = k < nz ? k + 1 : k, kb = ka - 1;
    tend[2 * st + k] = P(P_WSUBS, k) * ((th[ka] + P(P_THREF, ka)) - (th[kb] + P(P_THREF, kb))) * P(P_RDZN, ka);
  }
  if (q)
    for (int n = 0; n < s.nq; ++n) {
      const double* qp = olz + (3 + n) * st;
      const int ka = k < nz ? k + 1 : k, kb = ka - 1;
      tend[(3 + n) * st + k] = P(P_WSUBS, k) * (qp[ka] - qp[kb]) * P(P_RDZN, ka);
    }
}

int launch_subsidence_tendencies(const Scalars& s, const double* olz, double* tend, bool flow_theta, bool q,
                                 cudaStream_t st) {
  const int n = s.nz - 1;
  k_subsidence_tendencies<<<(n + 127) / 128, 128, 0, st>>>(s, olz, tend, flow_theta ? 1 : 0, q ? 1 : 0);
  return 1;
}

}  // namespace mgpu
