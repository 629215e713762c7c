// Momentum of the contracted build's centred step, shared-memory tiled: Piacsek-Williams advection
// (or the TVD sources of tvd_fast.cuh), viscosity, coriolis, buoyancy, damping, subsidence and
// stepfields of u, v, w (models with the iterative pressure solver keep k_f_momentum_tiled, see
// Scalars::krylov).
//
// The kernel it replaces was bound by shared-memory loads (84 eight-byte loads per point, 53% of the
// shared-memory pipe with 16 warps per SM).  Here
//  * every viscous stress is formed once, by the thread of its cell, and read by its neighbours from
//    a table -- tau12 had been formed three times per point, the other four twice;
//  * what a level shares with the one below (its own values and sums in the column, the stresses
//    through the face below) is carried up in registers;
//  * the reference density cancels (Boussinesq: rho = rhon on every level);
//  * the buoyancy of a level is formed once, from the q fields that have a weight, loaded a whole
//    level before it is used (used at once, those loads held the warps up: 0.282 against 0.254 ms
//    with two barriers a level).
// 256 x 256 x 128: FP64 0.275 -> 0.246 ms (738 MB, 0.113 ms), FP32 0.170 -> 0.151 ms; moist
// 512 x 512 x 160: 1.78 -> 1.15 and 1.02 -> 0.71 ms; 1024 x 1024 x 200 with five q fields, FP32:
// 7.07 -> 3.40 ms.  What is left in FP64 is latency with 16 warps per SM (128 registers, 90 KB): copies in
// flight, shared-memory loads and a barrier a level (45% of the issue slots, 58% of the shared-memory
// pipe); FP32 issues in 86% of its slots.
// Sizes that no tile divides run here too: 360 x 300 x 81 in FP64 took 1.67 ms in the point kernel
// for momentum and theta, now 0.28 and 0.28 ms.
#pragma once

namespace mgpu {
namespace KVARIANT {
namespace momf {

using tvdf::CN;
using tvdf::CW;
using tvdf::G;
using tvdf::NT;
using tvdf::PlaneStager;
using tvdf::TY;
using tiled::HY;
using tiled::TX;

enum { L_T1, L_T2, L_D1, L_D2, L_RDZ, L_RDZN, L_GWX, L_GWY, L_N };  // level constants (RDZN of k+1)
constexpr int RL = 4;
// levels k, k+1 and the one in flight; vis also k-1
constexpr int RP = 3, RVIS = 4;
template <typename T>
constexpr size_t smem_bytes() {
  return sizeof(T) * ((size_t)(6 * RP + RVIS) * G<T>::PLANE + (size_t)RL * L_N + (size_t)10 * CN);
}
template <typename T>
constexpr int ctas() { return sizeof(T) == 4 ? 4 : 2; }

template <typename T, bool TVD>
__global__ void __launch_bounds__(NT, ctas<T>()) k_f_momentum(const __grid_constant__ Scalars s,
                                                             const __grid_constant__ DevState<T> d, int kchunk) {
  using Gt = G<T>;
  constexpr int PL = Gt::PLANE, PW = Gt::PW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const rU = reinterpret_cast<T*>(smem_raw);
  T* const rV = rU + RP * PL;
  T* const rW = rV + RP * PL;
  T* const rZU = rW + RP * PL;
  T* const rZV = rZU + RP * PL;
  T* const rZW = rZV + RP * PL;
  T* const rVIS = rZW + RP * PL;
  T* const rL = rVIS + RVIS * PL;
  // the level's stresses: tau11, tau22 at the cells, tau12 at their upper right corners, tau13 and
  // tau23 on their right and upper sides
  // (two buffers, alternating with the level: see the loop)
  T* t11 = rL + RL * L_N;
  T* t_next = t11 + 5 * CN;
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TY;
  const int nz = s.nz;
  const int kb = 2 + (int)blockIdx.z * kchunk;
  const int ke = min(nz, kb + kchunk - 1);
  const long long plane = s.plane;
  const bool act = i0 + tx < s.nx && j0 + ty < s.ny;
  const int i = PlaneStager<T>::wrap(i0 + tx, s.nx), j = PlaneStager<T>::wrap(j0 + ty, s.ny);
  const int co = (ty + HY) * PW + (tx + Gt::V), own = (ty + 1) * CW + tx + 1;
  const T cx = (T)s.cx, cy = (T)s.cy;
  const bool vd = s.use_vd != 0;

  int l_at = 0;
  const bool l_thread = ty == TY - 1 && tx < L_N;
  if (l_thread) {
    const int ids[L_N] = {P_TZC1, P_TZC2, P_TZD1, P_TZD2, P_RDZ, P_RDZN, P_GWX, P_GWY};
    int id = 0;
#pragma unroll
    for (int q = 0; q < L_N; ++q)
      if (tx == q) id = ids[q];
    l_at = id * (nz + 2) + (tx == L_RDZN ? 1 : 0);
  }
  auto level_const = [&](int kk) { return (T)__ldg(s.prof + l_at + kk); };

  PlaneStager<T> sg;
  sg.init(s, j0, i0, tid);
  auto stage = [&](int kk) {
    const int o = (kk % RP) * PL;
    const long long lv = (long long)(kk - 1) * plane;
    sg.copy(rU + o, d.u + lv);
    sg.copy(rV + o, d.v + lv);
    sg.copy(rW + o, d.w + lv);
    if (vd) {
      sg.copy(rZU + o, d.zu + lv);
      sg.copy(rZV + o, d.zv + lv);
      sg.copy(rZW + o, d.zw + lv);
      sg.copy(rVIS + (kk % RVIS) * PL, d.vis + lv);
    }
  };
  for (int kk = kb; kk <= kb + 2 && kk <= min(nz, ke + 1); ++kk) stage(kk);
  if (vd) sg.copy(rVIS + ((kb - 1) % RVIS) * PL, d.vis + (long long)(kb - 2) * plane);
  if (l_thread)
    for (int kk = kb; kk <= kb + 1 && kk <= nz; ++kk) rL[(kk & (RL - 1)) * L_N + tx] = level_const(kk);
  const T dtm_x2 = (T)(2.0 * s.dtm);
  const long long col = (long long)j * s.nx + i;
  // Buoyancy of a level: half the weighted sum sw(k) takes from each of levels k and k+1; with
  // s.bmean the horizontal means are taken out (see buoyancy_point).  The values are loaded at the
  // top of a level and weighed at its end, so that no load is waited for.  Only vapour and liquid
  // (q fields 0 and 1) have a weight.
  const T bco = (T)0.5 * (T)__ldg(s.prof + P_BUOY_CO * (nz + 2) + 2);
  const bool b_th = !s.passive_th, b_q0 = !s.passive_q && s.nq > 0 && s.cq[0] != 0.0,
             b_q1 = !s.passive_q && s.nq > 1 && s.cq[1] != 0.0;
  const T w_q0 = (T)(0.5 * s.G * s.cq[0]), w_q1 = (T)(0.5 * s.G * s.cq[1]);
  struct Raw {
    T th, q0, q1;
  };
  auto load_raw = [&](long long o) {
    return Raw{b_th ? __ldg(d.th + o) : (T)0.0, b_q0 ? __ldg(d.q[0] + o) : (T)0.0, b_q1 ? __ldg(d.q[1] + o) : (T)0.0};
  };
  auto buoyancy = [&](int kk, const Raw& r) {
    T a = r.th, b = r.q0, c = r.q1;
    if (s.bmean) {
      a = a - (T)s.bmean[kk];
      if (b_q0) b = b - (T)s.bmean[(nz + 2) + kk];
      if (b_q1) c = c - (T)s.bmean[2 * (nz + 2) + kk];
    }
    T r0 = b_th ? bco * a : (T)0.0;
    if (b_q0) r0 = r0 + w_q0 * b;
    if (b_q1) r0 = r0 + w_q1 * c;
    return r0;
  };
  // values of level kb-1 and the stresses through the face below level kb, from global memory
  const int ip = i + 1 == s.nx ? 0 : i + 1, jp = j + 1 == s.ny ? 0 : j + 1;
  const long long lvm = (long long)(kb - 2) * plane, lv0 = lvm + plane;
  const long long ce = (long long)j * s.nx + ip, cn = (long long)jp * s.nx + i;
  T ud = __ldg(d.u + lvm + col), vdn = __ldg(d.v + lvm + col), wd = __ldg(d.w + lvm + col);
  T wxd = wd + __ldg(d.w + lvm + ce), wyd = wd + __ldg(d.w + lvm + cn);
  T t13d = (T)0.0, t23d = (T)0.0, t33 = (T)0.0;
  if (vd) {
    const T rz = (T)__ldg(s.prof + P_RDZN * (nz + 2) + kb), vm = __ldg(d.vis + lvm + col);
    const T zum = __ldg(d.zu + lvm + col), zvm = __ldg(d.zv + lvm + col), zwm = __ldg(d.zw + lvm + col);
    t13d = (T)0.5 * (vm + __ldg(d.vis + lvm + ce)) *
           ((__ldg(d.zu + lv0 + col) - zum) * rz + (__ldg(d.zw + lvm + ce) - zwm) * cx);
    t23d = (T)0.5 * (vm + __ldg(d.vis + lvm + cn)) *
           ((__ldg(d.zw + lvm + cn) - zwm) * cy + (__ldg(d.zv + lv0 + col) - zvm) * rz);
    t33 = (__ldg(d.vis + lv0 + col) + vm) * (__ldg(d.zw + lv0 + col) - zwm) * (T)__ldg(s.prof + P_RDZ * (nz + 2) + kb);
    if (kb == 2 && act) {
      // level 1: the sources are zero there (stepfields zeroes them)
      d.zu_n[col] = (T)s.ugal + zum;
      d.zv_n[col] = (T)s.vgal + zvm;
      d.zw_n[col] = zwm;
    }
  } else if (kb == 2 && act) {
    d.zu_n[col] = (T)s.ugal + d.zu[col];
    d.zv_n[col] = (T)s.vgal + d.zv[col];
    d.zw_n[col] = d.zw[col];
  }
  T blo = buoyancy(kb, load_raw(lv0 + col));
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  int s0 = (kb % RP) * PL, s1 = ((kb + 1) % RP) * PL, s2 = ((kb + 2) % RP) * PL;
  int vm_ = ((kb - 1) % RVIS) * PL, v0_ = (kb % RVIS) * PL, v1_ = ((kb + 1) % RVIS) * PL, v2_ = ((kb + 2) % RVIS) * PL;
  T u0 = rU[s0 + co], v0 = rV[s0 + co], w0 = rW[s0 + co];
  T pnext = l_thread && kb + 2 <= min(nz, ke + 1) ? level_const(kb + 2) : (T)0.0;
  long long lev = lv0;
  const unsigned sa = (unsigned)__cvta_generic_to_shared(rU + sg.soff);
  long long go = lev + 3 * plane + sg.goff;  // this thread's chunk of level k+3
  for (int k = kb; k <= ke; ++k, lev += plane, go += plane) {
    T *const t22 = t11 + CN, *const t12 = t22 + CN, *const t13 = t12 + CN, *const t23 = t13 + CN;
    // (loaded a level ahead; level k+1 reads it after this level's barrier)
    if (l_thread && k + 2 <= min(nz, ke + 1)) rL[((k + 2) & (RL - 1)) * L_N + tx] = pnext;
    if (l_thread && k + 3 <= min(nz, ke + 1)) pnext = level_const(k + 3);
    const long long o = lev + col;
    const bool in = k < nz;
    const Raw raw = in ? load_raw(o + plane) : Raw{(T)0.0, (T)0.0, (T)0.0};
    T tu = (T)0.0, tv = (T)0.0, tw = (T)0.0;
    if constexpr (TVD) {
      tu = __ldg(d.su + o);
      tv = __ldg(d.sv + o);
      tw = __ldg(d.sw + o);
    }
    const T* L = rL + (k & (RL - 1)) * L_N;
    const T *pU = rU + s0 + co, *pV = rV + s0 + co, *pW = rW + s0 + co;
    const T *qU = rU + s1 + co, *qV = rV + s1 + co;
    T su, sv, sw;
    // sums of neighbours that advection and coriolis share
    const T um = pU[-1], vs = pV[-PW];
    const T vx = v0 + pV[1], vxs = vs + pV[1 - PW], uy = u0 + pU[PW], uym = um + pU[PW - 1];
    const T wx = w0 + pW[1], wy = w0 + pW[PW];
    T uu = (T)0.0, vu = (T)0.0, wu = (T)0.0;  // level k+1
    if (in) {
      uu = qU[0];
      vu = qV[0];
      wu = rW[s1 + co];
    }
    if constexpr (TVD) {
      su = sv = sw = (T)0.0;  // added at the end
    } else {
      const T tcx = (T)s.tcx, tcy = (T)s.tcy;
      const T up = pU[1], us = pU[-PW], un = pU[PW], vm = pV[-1], vp = pV[1], vn = pV[PW];
      su = tcx * (um * (u0 + um) - up * (u0 + up)) + tcy * (us * vxs - un * vx) + L[L_T1] * ud * wxd;
      sv = tcy * (vs * (v0 + vs) - vn * (v0 + vn)) + tcx * (vm * uym - vp * uy) + L[L_T1] * vdn * wyd;
      sw = (T)0.0;
      if (in) {
        su = su - L[L_T2] * uu * wx;
        sv = sv - L[L_T2] * vu * wy;
        sw = L[L_D1] * wd * (w0 + wd) - L[L_D2] * wu * (w0 + wu);
        sw = sw + tcx * (pW[-1] * (um + qU[-1]) - pW[1] * (u0 + uu));
        sw = sw + tcy * (pW[-PW] * (vs + qV[-PW]) - pW[PW] * (v0 + vu));
      }
    }
    if (s.coriolis) {
      const T f = (T)s.fcoriol;
      su = su + f * ((T)0.25 * (vx + vxs) + (T)s.vgal - L[L_GWY]);
      sv = sv - f * ((T)0.25 * (uy + uym) + (T)s.ugal - L[L_GWX]);
    }
    T zu = (T)0.0, zv = (T)0.0, zw = (T)0.0, va = (T)0.0, m11 = (T)0.0, m22 = (T)0.0, m12 = (T)0.0, m13 = (T)0.0,
      m23 = (T)0.0, t33u = (T)0.0;
    if (vd) {
      const T *pZU = rZU + s0, *pZV = rZV + s0, *pZW = rZW + s0, *pA = rVIS + v0_, *pB = rVIS + vm_;
      // vis(k) + vis(k-1) of the cell at offset c, and the stresses of that cell
      auto vsum = [&](int c) { return pA[c] + pB[c]; };
      auto tau12 = [&](int c, T v4) {
        return (T)0.125 * v4 * ((pZU[c + PW] - pZU[c]) * cy + (pZV[c + 1] - pZV[c]) * cx);
      };
      auto tau13 = [&](int c, T z) {
        return (T)0.5 * (pA[c] + pA[c + 1]) * ((rZU[s1 + c] - z) * L[L_RDZN] + (pZW[c + 1] - pZW[c]) * cx);
      };
      auto tau23 = [&](int c, T z) {
        return (T)0.5 * (pA[c] + pA[c + PW]) * ((pZW[c + PW] - pZW[c]) * cy + (rZV[s1 + c] - z) * L[L_RDZN]);
      };
      zu = pZU[co];
      zv = pZV[co];
      zw = pZW[co];
      va = vsum(co);
      m11 = va * (zu - pZU[co - 1]) * cx;
      m22 = va * (zv - pZV[co - PW]) * cy;
      m12 = tau12(co, (va + vsum(co + PW)) + (vsum(co + 1) + vsum(co + PW + 1)));
      if (in) {
        m13 = tau13(co, zu);
        m23 = tau23(co, zv);
        t33u = (rVIS[v1_ + co] + pA[co]) * (rZW[s1 + co] - zw) * rL[((k + 1) & (RL - 1)) * L_N + L_RDZ];
      }
      t11[own] = m11;
      t22[own] = m22;
      t12[own] = m12;
      t13[own] = m13;
      t23[own] = m23;
      // the stresses around the tile that its cells read: below (warp 0), above (1), left (2), right (3)
      if (ty == 0) {
        const int c = (HY - 1) * PW + tx + Gt::V;
        t12[tx + 1] = tau12(c, (vsum(c) + vsum(c + PW)) + (vsum(c + 1) + vsum(c + PW + 1)));
        t23[tx + 1] = in ? tau23(c, pZV[c]) : (T)0.0;
      } else if (ty == 1) {
        const int c = (HY + TY) * PW + tx + Gt::V;
        t22[(TY + 1) * CW + tx + 1] = vsum(c) * (pZV[c] - pZV[c - PW]) * cy;
      } else if (ty == 2 && tx < TY) {
        const int c = (HY + tx) * PW + Gt::V - 1;
        t12[(tx + 1) * CW] = tau12(c, (vsum(c) + vsum(c + PW)) + (vsum(c + 1) + vsum(c + PW + 1)));
        t13[(tx + 1) * CW] = in ? tau13(c, pZU[c]) : (T)0.0;
      } else if (ty == 3 && tx < TY) {
        const int c = (HY + tx) * PW + Gt::V + TX;
        t11[(tx + 1) * CW + TX + 1] = vsum(c) * (pZU[c] - pZU[c - 1]) * cx;
      }
    } else if (act) {
      zu = d.zu[o];
      zv = d.zv[o];
      zw = d.zw[o];
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    // The stresses of the level are known, no plane of it is read below and level k+2 has landed: one
    // barrier a level.  (A thread ahead writes the next level's stresses to the other buffer.)
    if (k + 3 <= min(nz, ke + 1)) {
      const unsigned a = sa + (unsigned)(sizeof(T) * s0);
      constexpr unsigned RB = sizeof(T) * RP * PL;
      sg.copy_to(a, d.u + go);
      sg.copy_to(a + RB, d.v + go);
      sg.copy_to(a + 2 * RB, d.w + go);
      if (vd) {
        sg.copy_to(a + 3 * RB, d.zu + go);
        sg.copy_to(a + 4 * RB, d.zv + go);
        sg.copy_to(a + 5 * RB, d.zw + go);
        sg.copy_to(sa + 6 * RB + (unsigned)(sizeof(T) * vm_), d.vis + go);
      }
    }
    if (vd) {
      su = su + (t11[own + 1] - m11) * cx + (m12 - t12[own - CW]) * cy + (m13 - t13d) * L[L_RDZ];
      sv = sv + (m12 - t12[own - 1]) * cx + (t22[own + CW] - m22) * cy + (m23 - t23d) * L[L_RDZ];
      if (in) {
        sw = sw + (m13 - t13[own - 1]) * cx + (m23 - t23[own - CW]) * cy + (t33u - t33) * L[L_RDZN];
        t33 = t33u;
      }
      t13d = m13;
      t23d = m23;
    }
    const T bhi = in ? buoyancy(k + 1, raw) : (T)0.0;
    if (in) sw = sw + (blo + bhi);
    if constexpr (TVD) {
      su = su + tu;
      sv = sv + tv;
      sw = sw + tw;
    }
    if (s.damping || s.subs_th) {
      const Prof<T> P = prof<T>(s);
      if (s.damping) damping_flow_point<T>(s, P, k, zu, zv, zw, su, sv, sw);
      if (s.subs_th) subsidence_flow_point<T>(s, P, view<T>(d.zu, s), view<T>(d.zv, s), k, j, i, su, sv);
    }
    if (act) {
      d.zu_n[o] = (T)s.ugal + zu + dtm_x2 * su;
      d.zv_n[o] = (T)s.vgal + zv + dtm_x2 * sv;
      d.zw_n[o] = zw + dtm_x2 * sw;
    }
    ud = u0; vdn = v0; wd = w0;
    u0 = uu; v0 = vu; w0 = wu;
    wxd = wx; wyd = wy;
    blo = bhi;
    int q = s0;
    s0 = s1; s1 = s2; s2 = q;
    q = vm_;
    vm_ = v0_; v0_ = v1_; v1_ = v2_; v2_ = q;
    T* const t = t11;
    t11 = t_next;
    t_next = t;
  }
}

template <typename T>
static int launch(const Scalars& s, DevState<T>& d, cudaStream_t st) {
  const size_t smem = smem_bytes<T>();
  static LaunchTable table;
  const LaunchLimits lim =
      launch_limits(table, {(const void*)k_f_momentum<T, false>, (const void*)k_f_momentum<T, true>}, NT, smem);
  const int gx = (s.nx + TX - 1) / TX, gy = (s.ny + TY - 1) / TY, levels = s.nz - 1;
  const int nc = s.level_chunks > 0 ? s.level_chunks : tvdf::choose_chunks(gx * gy, lim.occ, lim.nsm, levels);
  const int kc = (levels + nc - 1) / nc;
  const dim3 grid(gx, gy, (levels + kc - 1) / kc);
  if (s.tvd_flow) k_f_momentum<T, true><<<grid, NT, smem, st>>>(s, d, kc);
  else k_f_momentum<T, false><<<grid, NT, smem, st>>>(s, d, kc);
  return 1;
}

}  // namespace momf
}  // namespace KVARIANT
}  // namespace mgpu
