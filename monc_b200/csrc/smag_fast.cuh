// Subgrid pass of the contracted build: Smagorinsky of levels 2 .. nz-1, zero at nz, and lower_bc on
// level 1 in one launch, any horizontal size (models with the iterative pressure solver keep
// k_f_smag_tiled, see Scalars::krylov).
//
// The horizontal shear of a cell sums four squared corner terms and the vertical shears two squared
// side terms each: a thread forms the corner and sides of its own cell and reads the others from a
// table, where the kernel this replaces formed all eight per point (27 shared-memory loads, 293
// instructions).  Tables alternate between two buffers, so that one barrier a level does: after it
// the planes of the level are no longer read and the next copies start.  The Richardson number's
// fields are loaded a level before they are used.  lower_bc takes the blocks of the first z index,
// beside the others.
// 256 x 256 x 128, lower_bc included: FP64 0.138 -> 0.124 ms (403 MB, 0.061 ms), FP32 0.098 -> 0.086 ms;
// moist 512 x 512 x 160: 0.864 -> 0.749 and 0.553 -> 0.489 ms; 360 x 300 x 81 in FP64, which no
// tile divides, 0.228 (point kernel) -> 0.153 ms.  Three blocks an SM in FP64 leave 80 registers, of which
// the moist form spills 20 bytes; four in FP32 (64) none.  FP64 issues in 58% of the slots and waits for the
// copies and direct loads with 23 warps per SM; FP32 issues in 77%.
#pragma once

namespace mgpu {
namespace KVARIANT {
namespace smagf {

using tvdf::CN;
using tvdf::CW;
using tvdf::G;
using tvdf::NT;
using tvdf::PlaneStager;
using tvdf::TY;
using tiled::HY;
using tiled::TX;

// level constants (RDZ and RDZN of k+1), the moist Richardson number's from L_QSAT on
enum { L_RDZ, L_RDZN, L_RNSQ, L_DTH, L_BUOY, L_QSAT, L_DQ, L_RPR, L_FAC, L_PR, L_THR, L_THR1, L_TREF, L_TST, L_TOFF, L_N };
constexpr int RL = 4;
constexpr int RUV = 2, RW = 3;  // planes of u, v (k+1 and the one in flight) and w (also k)
template <typename T>
constexpr size_t smem_bytes() {
  return sizeof(T) * ((size_t)(2 * RUV + RW) * G<T>::PLANE + (size_t)RL * L_N + (size_t)6 * CN);
}
template <typename T>
constexpr int ctas() { return sizeof(T) == 4 ? 4 : 3; }

// the staged level constants as a profile accessor of level k (k+1 where the code asks for it)
template <typename T>
struct LevelProf {
  const T* c;
  int k;
  __device__ __forceinline__ T operator()(int id, int kk) const {
    switch (id) {
      case P_RDZN: return c[L_RDZN];
      case P_RNEUTML_SQ: return c[L_RNSQ];
      case P_DTHREF: return c[L_DTH];
      case P_BUOY_CO: return c[L_BUOY];
      case P_QSAT: return c[L_QSAT];
      case P_DQSATDT: return c[L_DQ];
      case P_RPREFRCP: return c[L_RPR];
      case P_QSATFAC: return c[L_FAC];
      case P_PREFRCP: return c[L_PR];
      case P_THREF: return kk == k ? c[L_THR] : c[L_THR1];
      case P_TREF: return c[L_TREF];
      case P_TSTARPR: return c[L_TST];
      default: return c[L_TOFF];
    }
  }
};

// vis and diff from the strain rate and X = ri ssq (smagorinsky_from_strain's contracted form)
template <typename T>
__device__ __forceinline__ void stability(const Scalars& s, T rn, T ssq, T X, T& vis, T& diff) {
  if (X <= (T)0.0) {
    vis = rn * sqrt(ssq - (T)s.subc * X);
    diff = rn * ((T)s.suba * sqrt(ssq - (T)s.subb * X));
    return;
  }
  const T ri = X / ssq;
  vis = diff = (T)0.0;
  if (ri < (T)s.ric) {
    T t = (T)1. - ri * (T)s.ricinv;
    t = t * t;
    const T m = (t * t) * (rn * sqrt(ssq));
    vis = m * ((T)1. - (T)s.subh * ri);
    diff = m * ((T)s.suba * ((T)1. - (T)s.subg * ri));
  }
}

template <typename T>
__device__ __noinline__ void lower_bc_block(const Scalars& s, const DevState<T>& d, int j, int i) {
  const Prof<T> P = prof<T>(s);
  const bool fwd = s.forward;
  const View<T> zus = view<T>(d.zu, s), zua = view<T>(fwd ? d.u : d.zu, s), zva = view<T>(fwd ? d.v : d.zv, s);
  T* tha = fwd ? d.th : d.zth;
  View<T> qv;
  T* qa = nullptr;
  if (s.nq > 0) { qa = fwd ? d.q[s.iqv] : d.zq[s.iqv]; qv = view<T>(qa, s); }
  T vis1, diff1, th1, qv1;
  lower_bc_column<T>(s, P, zus, zua, zva, view<T>(tha, s), s.nq > 0 ? &qv : nullptr, j, i, vis1, diff1, th1, qv1);
  const long long o = lin(s, 1, j, i);
  d.vis[o] = vis1;
  d.diff[o] = diff1;
  tha[o] = th1;
  if (qa) qa[o] = qv1;
}

template <typename T, bool MOIST>
__global__ void __launch_bounds__(NT, ctas<T>()) k_f_smag(const __grid_constant__ Scalars s,
                                                         const __grid_constant__ DevState<T> d, int kchunk) {
  using Gt = G<T>;
  constexpr int PL = Gt::PLANE, PW = Gt::PW;
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TY;
  const bool act = i0 + tx < s.nx && j0 + ty < s.ny;
  if (blockIdx.z == 0) {
    if (act) lower_bc_block<T>(s, d, j0 + ty, i0 + tx);
    return;
  }
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const rU = reinterpret_cast<T*>(smem_raw);
  T* const rV = rU + RUV * PL;
  T* const rW = rV + RUV * PL;
  T* const rL = rW + RW * PL;
  T* const tab = rL + RL * L_N;  // two buffers of: corner terms of level k+1, x sides and y sides of level k
  const int nz = s.nz;
  const int kb = 2 + ((int)blockIdx.z - 1) * kchunk;
  const int ke = min(nz - 1, kb + kchunk - 1);
  const long long plane = s.plane;
  const bool fwd = s.forward;
  const int i = PlaneStager<T>::wrap(i0 + tx, s.nx), j = PlaneStager<T>::wrap(j0 + ty, s.ny);
  const int co = (ty + HY) * PW + (tx + Gt::V), own = (ty + 1) * CW + tx + 1;
  const T* const gu = fwd ? d.u : d.zu;
  const T* const gv = fwd ? d.v : d.zv;
  const T* const gw = fwd ? d.w : d.zw;
  const T cx = (T)s.cx, cy = (T)s.cy;

  int l_at = 0;
  const bool l_thread = ty == TY - 1 && tx < L_N;
  if (l_thread) {
    const int ids[L_N] = {P_RDZ,  P_RDZN,   P_RNEUTML_SQ, P_DTHREF,  P_BUOY_CO, P_QSAT, P_DQSATDT, P_RPREFRCP,
                          P_QSATFAC, P_PREFRCP, P_THREF,  P_THREF, P_TREF, P_TSTARPR, P_TOFF};
    int id = 0;
#pragma unroll
    for (int q = 0; q < L_N; ++q)
      if (tx == q) id = ids[q];
    l_at = id * (nz + 2) + (tx == L_RDZ || tx == L_RDZN || tx == L_THR1 ? 1 : 0);
  }
  auto level_const = [&](int kk) { return (T)__ldg(s.prof + l_at + kk); };

  PlaneStager<T> sg;
  sg.init(s, j0, i0, tid);
  auto stage_w = [&](int kk) { sg.copy(rW + (kk % RW) * PL, gw + (long long)(kk - 1) * plane); };
  auto stage = [&](int kk) {
    const int o = (kk % RUV) * PL;
    const long long lv = (long long)(kk - 1) * plane;
    sg.copy(rU + o, gu + lv);
    sg.copy(rV + o, gv + lv);
    stage_w(kk);
  };
  stage_w(kb);
  stage(kb + 1);
  if (kb + 2 <= min(nz, ke + 1)) stage(kb + 2);
  if (l_thread)
    for (int kk = kb; kk <= min(nz, kb + 1); ++kk) rL[(kk & (RL - 1)) * L_N + tx] = level_const(kk);
  const long long col = (long long)j * s.nx + i;
  if (ke == nz - 1 && act) {
    d.vis[(long long)(nz - 1) * plane + col] = (T)0.0;
    d.diff[(long long)(nz - 1) * plane + col] = (T)0.0;
  }
  // the fields of the Richardson number: theta of the current state (dry) or theta, vapour and
  // liquid of the advected one (moist)
  const T* const g_th = MOIST ? (fwd ? d.th : d.zth) : d.th;
  const T* const g_qv = MOIST ? (fwd ? d.q[s.iqv] : d.zq[s.iqv]) : nullptr;
  const T* const g_ql = MOIST ? (fwd ? d.q[s.iql] : d.zq[s.iql]) : nullptr;
  T th0, th1, qv0 = (T)0.0, qv1 = (T)0.0, ql0 = (T)0.0, ql1 = (T)0.0;
  const long long lvb = (long long)(kb - 1) * plane + col;
  th0 = __ldg(g_th + lvb);
  th1 = __ldg(g_th + lvb + plane);
  if constexpr (MOIST) {
    qv0 = __ldg(g_qv + lvb);
    qv1 = __ldg(g_qv + lvb + plane);
    ql0 = __ldg(g_ql + lvb);
    ql1 = __ldg(g_ql + lvb + plane);
  }
  // the parts of level kb from global memory; the border threads (below the tile: warp 0; to its left
  // and at its lower left corner: warp 1) keep u, v of their cell from level to level
  StrainLevel<T> lo = strain_level<T>(s, prof<T>(s), view<T>(gu, s), view<T>(gv, s), view<T>(gw, s), kb, j, i);
  T u0 = __ldg(gu + lvb), v0 = __ldg(gv + lvb), w0 = __ldg(gw + lvb);
  T b0 = (T)0.0;
  int bco = 0, bcell = 0;
  const bool below = ty == 0, left = ty == 1 && tx <= TY;  // lane TY of warp 1: the corner cell
  if (below) {
    bco = (HY - 1) * PW + tx + Gt::V;
    bcell = tx + 1;
    b0 = __ldg(gv + (long long)(kb - 1) * plane + (long long)PlaneStager<T>::wrap(j0 - 1, s.ny) * s.nx + i);
  } else if (left) {
    const int r = tx == TY ? -1 : tx;
    bco = (HY + r) * PW + Gt::V - 1;
    bcell = (r + 1) * CW;
    b0 = __ldg(gu + (long long)(kb - 1) * plane + (long long)PlaneStager<T>::wrap(j0 + r, s.ny) * s.nx +
               PlaneStager<T>::wrap(i0 - 1, s.nx));
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  int su_ = ((kb + 1) % RUV) * PL, sw0 = (kb % RW) * PL, sw1 = ((kb + 1) % RW) * PL, sw2 = ((kb + 2) % RW) * PL;
  T* tc = tab;
  T* tn = tab + 3 * CN;
  long long lev = lvb;
  for (int k = kb; k <= ke; ++k, lev += plane) {
    const T* L = rL + (k & (RL - 1)) * L_N;
    const T *pU = rU + su_, *pV = rV + su_, *pW = rW + sw0;
    const T rdzn = L[L_RDZN];
    T th2 = (T)0.0, qv2 = (T)0.0, ql2 = (T)0.0;
    if (k + 2 <= nz) {
      th2 = __ldg(g_th + lev + 2 * plane);
      if constexpr (MOIST) {
        qv2 = __ldg(g_qv + lev + 2 * plane);
        ql2 = __ldg(g_ql + lev + 2 * plane);
      }
    }
    const bool pstage = l_thread && k + 2 <= ke;
    const T pnext = pstage ? level_const(k + 2) : (T)0.0;
    // corner at level k+1 and the sides at level k of the cell at plane offset c
    auto corner = [&](int c) { return sqr((pU[c + PW] - pU[c]) * cy + (pV[c + 1] - pV[c]) * cx); };
    auto side_x = [&](int c, T u, T w) { return sqr((pU[c] - u) * rdzn + (pW[c + 1] - w) * cx); };
    auto side_y = [&](int c, T v, T w) { return sqr((pW[c + PW] - w) * cy + (pV[c] - v) * rdzn); };
    const T un = pU[co], vn = pV[co], wn = rW[sw1 + co];
    const T c12 = corner(co), c13 = side_x(co, u0, w0), c23 = side_y(co, v0, w0);
    StrainLevel<T> hi;
    hi.a11 = sqr(un - pU[co - 1]);
    hi.a22 = sqr(vn - pV[co - PW]);
    hi.a33 = sqr((wn - w0) * L[L_RDZ]);
    tc[own] = c12;
    tc[CN + own] = c13;
    tc[2 * CN + own] = c23;
    if (below) {
      tc[bcell] = corner(bco);
      tc[2 * CN + bcell] = side_y(bco, b0, pW[bco]);
      b0 = pV[bco];
    } else if (left) {
      tc[bcell] = corner(bco);
      tc[CN + bcell] = side_x(bco, b0, pW[bco]);
      b0 = pU[bco];
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    // the planes of level k+1 (u, v) and k (w) are free: the copies two levels up start
    if (k + 3 <= min(nz, ke + 1)) {
      sg.copy(rU + su_, gu + (lev - col) + 3 * plane);
      sg.copy(rV + su_, gv + (lev - col) + 3 * plane);
      sg.copy(rW + sw0, gw + (lev - col) + 3 * plane);
    }
    hi.g12 = (tc[own - CW - 1] + tc[own - 1]) + (tc[own - CW] + c12);
    const T ssq = (T)s.cx2 * (hi.a11 + lo.a11) + (T)s.cy2 * (hi.a22 + lo.a22) + (lo.a33 + hi.a33) +
                  (T)0.5 * ((c13 + tc[CN + own - 1]) + (c23 + tc[2 * CN + own - CW])) + (T)0.125 * (lo.g12 + hi.g12) +
                  (T)s.smallp;
    lo = hi;
    T vis, diff;
    const LevelProf<T> P{L, k};
    const ColPair<T> TH{th0, th1, k}, QV{qv0, qv1, k}, QL{ql0, ql1, k};
    T X = (T)0.0;  // Richardson number times ssq
    if (!s.passive_th) {
      if constexpr (MOIST) X = moist_ri<T, ColPair<T>, LevelProf<T>, true>(s, P, ssq, TH, QV, QL, k, j, i);
      else X = (L[L_DTH] + th1 - th0) * rdzn * L[L_BUOY];
    }
    stability<T>(s, L[L_RNSQ], ssq, X, vis, diff);
    if (act) {
      d.vis[lev] = vis;
      d.diff[lev] = diff;
    }
    if (pstage) rL[((k + 2) & (RL - 1)) * L_N + tx] = pnext;
    u0 = un; v0 = vn; w0 = wn;
    th0 = th1; th1 = th2;
    qv0 = qv1; qv1 = qv2;
    ql0 = ql1; ql1 = ql2;
    su_ = PL - su_;
    const int q = sw0;
    sw0 = sw1; sw1 = sw2; sw2 = q;
    T* const t = tc;
    tc = tn;
    tn = t;
  }
}

template <typename T, bool MOIST>
static int launch_as(const Scalars& s, DevState<T>& d, cudaStream_t st) {
  const size_t smem = smem_bytes<T>();
  static LaunchTable table;
  const LaunchLimits lim = launch_limits(table, {(const void*)k_f_smag<T, MOIST>}, NT, smem);
  const int gx = (s.nx + TX - 1) / TX, gy = (s.ny + TY - 1) / TY, levels = s.nz - 2;
  const int nc = s.level_chunks > 0 ? s.level_chunks : tvdf::choose_chunks(gx * gy, lim.occ, lim.nsm, levels);
  const int kc = (levels + nc - 1) / nc;
  k_f_smag<T, MOIST><<<dim3(gx, gy, 1 + (levels + kc - 1) / kc), NT, smem, st>>>(s, d, kc);
  return 1;
}
template <typename T>
static int launch(const Scalars& s, DevState<T>& d, cudaStream_t st) {
  return !s.passive_q && s.nq > 1 ? launch_as<T, true>(s, d, st) : launch_as<T, false>(s, d, st);
}

}  // namespace smagf
}  // namespace KVARIANT
}  // namespace mgpu
