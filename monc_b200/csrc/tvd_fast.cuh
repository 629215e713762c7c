// TVD (ULTIMATE-QUICKEST) advection of the contracted build's centred step, shared-memory tiled
// (models with the iterative pressure solver keep the kernels of dycore_kernels.cuh, see
// Scalars::krylov).
//
// One kernel advects NS fields together -- theta alone, theta with vapour and liquid (and the
// saturation adjustment), groups of tracers, or one flow component on its dual grid (DIM 0, 1, 2) --
// and, for scalars, adds diffusion, damping and subsidence and steps them.  A CTA owns a tile of
// 32 x 8 columns and marches up a chunk of levels; planes with a halo of 2 points are staged a
// level ahead with cp.async.  Sizes that no tile divides are allowed: the staged planes wrap
// periodically past the domain's edge and the columns beyond it are computed and not stored.
//
// What bounds it is instruction issue (FP32: 88% of the slots) and in FP64, with 16 warps per SM, the
// shared-memory pipe (71%, three fields 60%; 56% of the issue slots), so the face formulas (ultimateflux.F90)
// are arranged for few instructions and are equal to tvd_face_x/y/z of dycore_device.cuh to rounding:
//  * upwind values are addressed, not selected: the sign of the velocity picks the upwind cell and
//    a direction, and three loads give fu, fc, fd;
//  * the limiter is taken on magnitudes relative to fc (see limit), without a division by fd - fu
//    and without a branch, so that the loads and chains of a level's faces overlap;
//  * what a cell contributes to the faces around it -- its sums of u, v, w for the gradient terms
//    and the reciprocal of its outflow Courant sum -- is formed once per cell and level and shared
//    through a table; positive parts are x + |x|, an addition with an operand modifier;
//  * the velocity part of a face is formed once for the NS fields;
//  * the vertical metrics come as four ready coefficients per level (P_TVC1P ..).
// Measured against the kernels of the separately rounded build's form (developed flow): theta at
// 256 x 256 x 128 0.373 -> 0.246 ms in FP64 and 0.250 -> 0.162 ms in FP32; theta, vapour and liquid
// at 512 x 512 x 160 5.78 -> 2.54 and 3.47 -> 1.35 ms; theta and five q fields at 1024 x 1024 x 200
// in FP32 36.6 -> 12.2 ms; u, v, w at 256 x 256 x 128 in FP64 1.12 -> 0.64 ms.  FP64 moves 537 MB
// for theta, 0.082 ms.
#pragma once

#include "reciprocal.cuh"

namespace mgpu {
namespace KVARIANT {
namespace tvdf {

using tiled::TX;
using tiled::HY;

// The border of a tile -- the cells around it, and the faces between those below and to the left of
// it and the tile -- is spread over the block: warps 0, 1 and 2 form the cells below, above and to
// the sides, warps 3 and 4 the faces.  A warp that had both held the others up at every barrier
// (theta, FP64, 256 x 256 x 128: 0.292 -> 0.277 ms).
constexpr int TY = 8, NT = TX * TY;
constexpr int CW = TX + 2, CN = (TY + 2) * CW;  // the table of cells, border included
template <typename T>
struct G {
  static constexpr int V = 16 / (int)sizeof(T);  // elements per 16-byte chunk = x halo width
  static constexpr int PW = TX + 2 * V, PH = TY + 2 * HY, PLANE = PW * PH;
  static constexpr int CPR = PW / V, NCH = CPR * PH;  // chunks per plane row and per plane
  static_assert(NCH <= NT && (PLANE * sizeof(T)) % 16 == 0, "one chunk per thread and plane");
};

// level constants staged per level (a ring of 4 levels)
enum { L_C1P, L_C2P, L_C1N, L_C2N, L_WS, L_CS, L_WDT, L_T1, L_T2, L_CZB, L_CZA, L_REX, L_PRE, L_PREFN, L_TOFF, L_N = 16 };
constexpr int RL = 4;

// ring depths: the advected fields need levels k-1 .. k+2 and the one in flight; the flow is only
// read to form the next level's cell table (w on its dual grid averages two levels)
template <int DIM>
struct Rings {
  static constexpr int UP = DIM == 2 ? 1 : 0;  // levels above k+1 the table of level k+1 reads
  static constexpr int RZ = 5, RF = 2 + UP, RD = DIM < 0 ? 3 : 0;
};
// Two copies of the face fluxes and cell tables, alternating with the level, make one barrier a level
// do (theta, FP64, 256 x 256 x 128: 0.277 -> 0.246 ms); three FP64 fields leave no room for them at two CTAs.
template <typename T, int NS>
constexpr int copies() { return sizeof(T) == 8 && NS == 3 ? 1 : 2; }
template <typename T, int NS, int DIM>
constexpr size_t smem_bytes() {
  typedef Rings<DIM> R;
  return sizeof(T) * ((size_t)(NS * R::RZ + 3 * R::RF + R::RD) * G<T>::PLANE + (size_t)RL * L_N +
                      copies<T, NS>() * ((size_t)4 * CN + (size_t)NS * (TY * (TX + 1) + (TY + 1) * TX) + TX + TY));
}
// Resident CTAs the registers are sized for.  FP64 at two CTAs (no spills) runs faster than at
// three with 80 registers and spills (0.292 against 0.326 ms for theta at 256 x 256 x 128); FP32
// fits 64 registers, and four CTAs beat three (0.171 against 0.188 ms), three beat two for three
// fields (1.48 against 1.64 ms at 512 x 512 x 160).
template <typename T, int NS, int DIM>
constexpr int ctas() {
  if (sizeof(T) == 4) return NS == 1 && DIM != 2 ? 4 : 3;  // (w's dual grid takes more registers)
  return 2;
}

template <typename T> struct Pair;
template <> struct Pair<double> { typedef double2 t; };
template <> struct Pair<float> { typedef float2 t; };

__device__ __forceinline__ int hi_word(double x) { return __double2hiint(x); }
__device__ __forceinline__ int hi_word(float x) { return __float_as_int(x); }
// x with its sign bit flipped when m is the sign mask 0x80000000 (unchanged for m = 0)
__device__ __forceinline__ double flip(double x, int m) { return __hiloint2double(__double2hiint(x) ^ m, __double2loint(x)); }
__device__ __forceinline__ float flip(float x, int m) { return __int_as_float(__float_as_int(x) ^ m); }
template <typename T> __device__ __forceinline__ bool negative(T x) { return hi_word(x) < 0; }

// max(0, x) by the sign bit
__device__ __forceinline__ double positive(double x) {
  const int h = __double2hiint(x), m = ~(h >> 31);
  return __hiloint2double(h & m, __double2loint(x) & m);
}
__device__ __forceinline__ float positive(float x) { return x > 0.0f ? x : 0.0f; }
// The limited face value for fc - fu = a, fd - fc = e, the unlimited face b less fc, and r1 = 1 / S
// - 1 of the upwind cell's outflow Courant sum S.  The limiter's max(a, min(b, a / S, fd - fu)) on
// magnitudes, less a: max(0, min(b, a r1, e)) in the direction of a, added to fc.  Where a and e
// differ in sign (no monotone profile: |curvature| >= |fd - fu|) that is 0 and the face is fc.
template <typename T>
__device__ __forceinline__ T limit(T fc, T a, T e, T b, T r1) {
  const int m = hi_word(a) & (int)0x80000000;
  T y = tmin<T>(flip(a, m) * r1, flip(e, m));
  y = positive(tmin<T>(flip(b, m), y));
  return fc + flip(y, m);
}

// what one cell contributes to its faces: us, vs, ws the scaled sums of u, v, w over the cell's two
// faces in each direction (gradient terms), r = 1 / (outflow Courant sum + 1e-30) - 1
template <typename T>
struct Cell {
  T us, vs, ws, r;
};
template <typename T>
struct CellScale {
  T kx8, ky8, hx, hy;  // 0.125 cx dt, 0.125 cy dt, 0.5 cx dt, 0.5 cy dt
};
template <typename T>
__device__ __forceinline__ Cell<T> make_cell(const CellScale<T>& c, T ws_c, T cs_c, T u, T um, T v, T vm, T w, T wm) {
  Cell<T> r;
  r.us = (u + um) * c.kx8;
  r.vs = (v + vm) * c.ky8;
  r.ws = (w + wm) * ws_c;
  // max(0, x) + |min(0, y)| = ((x + |x|) + (|y| - y)) / 2, the halves in the coefficients
  const T S = cs_c * ((w + fabs(w)) + (fabs(wm) - wm)) + c.hy * ((v + fabs(v)) + (fabs(vm) - vm)) +
              c.hx * ((u + fabs(u)) + (fabs(um) - um));
  r.r = rcp_newton(S + (T)1.e-30) - (T)1.0;
  return r;
}

// value at offset o of a staged flow plane p, on the dual grid of flow component DIM (DualFlow);
// pn is the plane above, top says that p is the top level
template <typename T, int DIM>
__device__ __forceinline__ T dual(const T* p, const T* pn, int o, bool top) {
  if constexpr (DIM == 0) return (T)0.5 * (p[o] + p[o + 1]);
  else if constexpr (DIM == 1) return (T)0.5 * (p[o] + p[o + G<T>::PW]);
  else if constexpr (DIM == 2) return top ? p[o] : (T)0.5 * (p[o] + pn[o]);
  else return p[o];
}

// One thread's share of staging a plane: one chunk of G<T>::V elements, copied as 16 bytes, or as
// two halves where a row is not a whole number of chunks (FP32 with nx not a multiple of 4) and
// the periodic wrap may fall inside a chunk.  The tile may reach past the domain: every index is
// taken modulo the row length and the row count.
template <typename T>
struct PlaneStager {
  int soff;
  int goff, goff2;  // element offsets inside a level
  bool on, halves;
  __device__ __forceinline__ static int wrap(int i, int n) {
    i %= n;
    return i < 0 ? i + n : i;
  }
  __device__ void init(const Scalars& s, int j0, int i0, int tid) {
    using Gt = G<T>;
    on = tid < Gt::NCH;
    const int c = on ? tid : 0;
    const int row = c / Gt::CPR, cc = c - row * Gt::CPR;
    soff = row * Gt::PW + cc * Gt::V;
    const int gj = wrap(j0 - HY + row, s.ny), gi = i0 - Gt::V + cc * Gt::V;
    halves = sizeof(T) == 4 && (s.nx & (Gt::V - 1)) != 0;
    goff = gj * s.nx + wrap(gi, s.nx);
    goff2 = gj * s.nx + wrap(gi + Gt::V / 2, s.nx);
  }
  // level pointer `lev` (the field's base plus whole levels) into the plane at `dst`
  __device__ __forceinline__ void copy(T* dst, const T* __restrict__ lev) const {
    copy_to((unsigned)__cvta_generic_to_shared(dst + soff), lev + goff);
  }
  // the same with this thread's offsets (soff, goff) already in the two addresses
  __device__ __forceinline__ void copy_to(unsigned a, const T* __restrict__ g) const {
    if (!on) return;
    if (sizeof(T) == 4 && halves) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(a), "l"(g) : "memory");
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(a + 8), "l"(g + (goff2 - goff)) : "memory");
    } else {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(a), "l"(g) : "memory");
    }
  }
};

template <typename T, int NS>
struct Job {
  const T *u, *v, *w, *diff;
  const T* zf[NS];   // the advected fields
  const T* f[NS];    // scalars: the state fields (th or q)
  T* out_f[NS];      // scalars: stepped state and z-field
  T* out_zf[NS];
  T* src;            // flow component: the advective source
  int row[NS];       // scalars: the field's row in the mean profiles (2 theta, 3 + n q(n))
  int first;         // the first field is theta (no clip; baroclinicity)
};

// the staged level constants as the profile accessor simplecloud reads
template <typename T>
struct CloudProf {
  const T* c;
  int k;
  const Scalars& s;
  __device__ __forceinline__ T operator()(int id, int kk) const {
    if (kk != k) return load_profile<T>(s, id, kk);
    return c[id == P_RPREFRCP ? L_REX : (id == P_PREFRCP ? L_PRE : (id == P_PREFN ? L_PREFN : L_TOFF))];
  }
};

// the column's own values at levels k-1, k, k+1 as a field accessor
template <typename T>
struct Col3 {
  T m, z, p;
  int k;
  __device__ __forceinline__ T operator()(int kk, int, int) const { return kk < k ? m : (kk == k ? z : p); }
};

template <typename T, int NS, bool CLOUD, int DIM>
__global__ void __launch_bounds__(NT, ctas<T, NS, DIM>()) k_f_tvd(const __grid_constant__ Scalars s,
                                                                 const __grid_constant__ Job<T, NS> job, int kchunk) {
  using Gt = G<T>;
  typedef Rings<DIM> R;
  typedef typename Pair<T>::t T2;
  constexpr int PL = Gt::PLANE, PW = Gt::PW;
  constexpr int NFX = TY * (TX + 1), NFY = (TY + 1) * TX;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const rF = reinterpret_cast<T*>(smem_raw);         // NS rings of RZ planes
  T* const rU = rF + NS * R::RZ * PL;
  T* const rV = rU + R::RF * PL;
  T* const rW = rV + R::RF * PL;
  T* const rD = rW + R::RF * PL;
  T* const rL = rD + R::RD * PL;                        // level constants
  // of each copy: cell tables (vs, ws) and (us, r), NS x x-face fluxes of columns i0-1 .. i0+TX-1, NS x
  // y-face fluxes of rows j0-1 .. j0+TY-1, v of the cells below the tile and u of those to its left
  constexpr bool DB = copies<T, NS>() == 2;
  constexpr int COPY = 4 * CN + NS * (NFX + NFY) + TX + TY;
  T* cur = rL + RL * L_N;             // the copy of level k
  T* nxt = DB ? cur + COPY : cur;     // and that of level k+1
  const int tid = threadIdx.x, lane = tid & 31;
  const int tx = lane, ty = tid >> 5;  // the warp's row
  const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TY;
  const int nz = s.nz;
  const int ktop = DIM == 2 ? nz - 1 : nz;  // the last level with a source
  const int kb = 2 + (int)blockIdx.z * kchunk;
  const int ke = min(nz, kb + kchunk - 1);
  const long long plane = s.plane;
  const bool act = i0 + tx < s.nx && j0 + ty < s.ny;
  // the column's own indices, wrapped into the domain for the threads beyond its edge
  const int i = PlaneStager<T>::wrap(i0 + tx, s.nx), j = PlaneStager<T>::wrap(j0 + ty, s.ny);
  const int co = (ty + HY) * PW + (tx + Gt::V);
  const int own = (ty + 1) * CW + tx + 1;
  // this thread's cell of the border (row hr of the cell table, column hc; none: hr < 0)
  int hr = -1, hc = lane + 1;
  if (ty == 0) hr = 0;
  else if (ty == 1) hr = TY + 1;
  else if (ty == 2 && lane < 2 * TY) { hr = lane % TY + 1; hc = lane < TY ? 0 : TX + 1; }
  const int bco = (hr - 1 + HY) * PW + (hc - 1 + Gt::V), bcell = hr * CW + hc;
  // the level constant this thread stages
  int l_at = 0;
  double l_scale = 0.0;
  const double dt_d = s.dtm * 2.0;
  const bool l_thread = ty == TY - 1 && lane < L_N;  // stages the level constants
  if (l_thread) {
    constexpr bool WM = DIM == 2;
    int id = P_RDZ, sh = 0;
    l_scale = 1.0;
    switch (lane) {
      case L_C1P: id = WM ? P_TWC1P : P_TVC1P; break;
      case L_C2P: id = WM ? P_TWC2P : P_TVC2P; break;
      case L_C1N: id = WM ? P_TWC1N : P_TVC1N; break;
      case L_C2N: id = WM ? P_TWC2N : P_TVC2N; break;
      case L_WS: id = WM ? P_RDZN : P_RDZ; sh = WM ? 1 : 0; l_scale = 0.125 * dt_d; break;
      case L_CS: id = WM ? P_RDZN : P_RDZ; l_scale = 0.5 * dt_d; break;
      case L_WDT: id = WM ? P_RDZ : P_RDZN; sh = 1; l_scale = dt_d; break;
      case L_T1: id = WM ? P_TZD1 : P_TZC1; l_scale = 4.0; break;
      case L_T2: id = WM ? P_TZD2 : P_TZC2; l_scale = 4.0; break;
      case L_CZB: id = P_CZB; break;
      case L_CZA: id = P_CZA; break;
      case L_REX: id = P_RPREFRCP; break;
      case L_PRE: id = P_PREFRCP; break;
      case L_PREFN: id = P_PREFN; break;
      case L_TOFF: id = sizeof(T) == 4 ? P_TC0 : P_THREF; break;
      default: l_scale = 0.0; break;
    }
    l_at = id * (nz + 2) + sh;
  }
  auto level_const = [&](int kk) { return (T)(l_scale * __ldg(s.prof + l_at + kk)); };

  PlaneStager<T> sg;
  sg.init(s, j0, i0, tid);
  T2 *tVW = reinterpret_cast<T2*>(cur), *tUR = tVW + CN;
  T* BV = cur + 4 * CN + NS * (NFX + NFY);
  const int k0 = kb == 2 ? 1 : kb - 2;
  // advected fields kb-2 .. kb+2 (level k in slot k mod RZ), flow and diff as many as their rings hold
  for (int kk = k0; kk <= kb + 2 && kk <= nz; ++kk) {
    T* dst = rF + (kk % R::RZ) * PL;
    const long long lv = (long long)(kk - 1) * plane;
#pragma unroll
    for (int n = 0; n < NS; ++n) sg.copy(dst + n * R::RZ * PL, job.zf[n] + lv);
  }
  auto stage_flow = [&](int kk) {
    const int o = (kk % R::RF) * PL;
    const long long lv = (long long)(kk - 1) * plane;
    sg.copy(rU + o, job.u + lv);
    sg.copy(rV + o, job.v + lv);
    sg.copy(rW + o, job.w + lv);
  };
  for (int kk = kb + 1; kk <= kb + 2 + R::UP && kk <= min(nz, ke + 1 + R::UP); ++kk) stage_flow(kk);
  if constexpr (DIM < 0)
    for (int kk = kb - 1; kk <= kb + 1 && kk <= ke; ++kk) sg.copy(rD + (kk % 3) * PL, job.diff + (long long)(kk - 1) * plane);
  if (l_thread)
    for (int kk = kb - 1; kk <= kb + 1 && kk <= nz; ++kk) rL[(kk & (RL - 1)) * L_N + lane] = level_const(kk);
  const T dtm_x2 = (T)dt_d;
  const T c1 = (T)(1.0 - 2.0 * s.tsmth), c2 = (T)s.tsmth;
  const long long col = (long long)j * s.nx + i;
  if constexpr (DIM < 0) {
    if (kb == 2 && act) {
      // level 1: zero source
#pragma unroll
      for (int n = 0; n < NS; ++n) {
        const T fv = job.f[n][col], zv = job.zf[n][col];
        T zn = zv;
        if ((n > 0 || !job.first) && zn < (T)0.0) zn = (T)0.0;
        job.out_zf[n][col] = (c1 * fv + c2 * zv) + c2 * zn;
        job.out_f[n][col] = zn;
      }
    }
  }
  CellScale<T> cs;
  const T cdx = (T)(s.cx * dt_d), cdy = (T)(s.cy * dt_d);
  cs.kx8 = (T)0.125 * cdx;
  cs.ky8 = (T)0.125 * cdy;
  cs.hx = (T)0.5 * cdx;
  cs.hy = (T)0.5 * cdy;
  const T cx = (T)s.cx, cy = (T)s.cy, r6 = (T)(1.0 / 6.0);

  // the first cells from global memory, while the copies are in flight: the own cell at kb-1 (for
  // the z face below the chunk) and at kb, the border cell at kb
  typedef DualFlow<T, View<T>, DIM < 0 ? 0 : DIM> GF;
  const View<T> gU = view<T>(job.u, s), gV = view<T>(job.v, s), gW = view<T>(job.w, s);
  auto gflow = [&](const View<T>& a, int kk, int jj, int ii) -> T {
    if constexpr (DIM < 0) return a(kk, jj, ii);
    else return GF{a, nz}(kk, jj, ii);
  };
  auto gcell = [&](int kk, int jj, int ii, T& u, T& v, T& w, T wm, T ws_c, T cs_c) {
    u = gflow(gU, kk, jj, ii);
    v = gflow(gV, kk, jj, ii);
    w = gflow(gW, kk, jj, ii);
    return make_cell<T>(cs, ws_c, cs_c, u, gflow(gU, kk, jj, ii - 1), v, gflow(gV, kk, jj - 1, ii), w, wm);
  };
  auto gconst = [&](int slot, int kk) -> T {
    constexpr bool WM = DIM == 2;
    if (slot == L_WS) return (T)(0.125 * dt_d * __ldg(s.prof + (WM ? P_RDZN : P_RDZ) * (nz + 2) + kk + (WM ? 1 : 0)));
    return (T)(0.5 * dt_d * __ldg(s.prof + (WM ? P_RDZN : P_RDZ) * (nz + 2) + kk));
  };
  T u0 = (T)0.0, v0 = (T)0.0, w0 = (T)0.0, fz_lo[NS];
  T bw = (T)0.0;  // w of the border cell
#pragma unroll
  for (int n = 0; n < NS; ++n) fz_lo[n] = (T)0.0;
  Cell<T> cm{}, c0{};
  T wlow = (T)0.0;
  const T ws0 = gconst(L_WS, kb), cs0 = gconst(L_CS, kb);
  if (kb > 2) {
    T um, vm;
    cm = gcell(kb - 1, j, i, um, vm, wlow, gflow(gW, kb - 2, j, i), gconst(L_WS, kb - 1), gconst(L_CS, kb - 1));
  } else {
    wlow = gflow(gW, 1, j, i);
  }
  c0 = gcell(kb, j, i, u0, v0, w0, wlow, ws0, cs0);
  tVW[own] = T2{c0.vs, c0.ws};
  tUR[own] = T2{c0.us, c0.r};
  if (hr >= 0) {
    const int bj = PlaneStager<T>::wrap(j0 - 1 + hr, s.ny), bi = PlaneStager<T>::wrap(i0 - 1 + hc, s.nx);
    T bu, bv;
    const Cell<T> cb = gcell(kb, bj, bi, bu, bv, bw, gflow(gW, kb - 1, bj, bi), ws0, cs0);
    tVW[bcell] = T2{cb.vs, cb.ws};
    tUR[bcell] = T2{cb.us, cb.r};
    if (hr == 0) BV[lane] = bv;
    if (hc == 0) BV[TX + lane] = bu;
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();

  // z-face flux above level kk from the plane offsets of kk-1 .. kk+2 (the column's own point) and
  // the cells of kk and kk+1
  auto z_face = [&](int kk, T w, int zm, int z0, int z1, int z2, T vsum, T usum, T rlo, T rhi, const T* L, T* out) {
    const bool neg = negative(w);
    const T cmod = fabs(w) * L[L_WDT], omc = (T)1.0 - cmod, opc = (T)1.0 + cmod;
    const T2 cc = *reinterpret_cast<const T2*>(L + (neg ? L_C1N : L_C1P));
    const T r = neg ? rhi : rlo;
    const int oc = co + (neg ? z1 : z0), od = co + (neg ? z0 : z1), ou = co + (neg ? z2 : zm);
    const int sy = negative(vsum) ? PW : -PW, sx = negative(usum) ? 1 : -1;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      const T* p = rF + n * R::RZ * PL;
      const T fc = p[oc], fd = p[od];
      // beyond the top the field goes on linearly
      const T fu = (neg && kk + 2 > nz) ? (T)2.0 * fc - fd : p[ou];
      const T a = fc - fu, e = fd - fc;
      T b = omc * ((T)0.5 * e - opc * (e * cc.x - a * cc.y));
      b = b - fabs(vsum) * (fc - p[oc + sy]) - fabs(usum) * (fc - p[oc + sx]);
      out[n] = w * limit<T>(fc, a, e, b, r);
    }
  };
  int zm = ((kb - 1) % R::RZ) * PL, z0 = (kb % R::RZ) * PL, z1 = ((kb + 1) % R::RZ) * PL, z2 = ((kb + 2) % R::RZ) * PL,
      z3 = ((kb + 3) % R::RZ) * PL;
  if (kb > 2) {
    T rhi = c0.r;
    if (kb == nz && w0 != (T)0.0)  // as below the top level in the loop
      rhi = make_cell<T>(cs, gconst(L_WS, kb), gconst(L_CS, kb), u0, gflow(gU, kb, j, i - 1), v0, gflow(gV, kb, j - 1, i),
                         (T)0.0, wlow).r;
    z_face(kb - 1, wlow, z3, zm, z0, z1, cm.vs + c0.vs, cm.us + c0.us, cm.r, rhi, rL + ((kb - 1) & (RL - 1)) * L_N, fz_lo);
  } else if constexpr (DIM == 2) {
    const GF IU{gU, nz}, IV{gV, nz}, IW{gW, nz};
    fz_lo[0] = wlow * tvd_face_z_bottom<T, GF, View<T>, Prof<T>, TvdMetricW>(s, prof<T>(s), IU, IV, IW,
                                                                            view<T>(job.zf[0], s), dtm_x2, j, i);
  }
  int dm = ((kb - 1) % 3) * PL, d0 = (kb % 3) * PL, d1 = ((kb + 1) % 3) * PL;
  int fo = ((kb + 1) % R::RF) * PL;             // slot of the flow at k+1
  long long lev = (long long)(kb - 1) * plane;  // offset of level k
  const unsigned sa = (unsigned)__cvta_generic_to_shared(rF + sg.soff);
  long long go = lev + sg.goff;
  auto stage_field = [&](int slot, long long off) {
#pragma unroll
    for (int n = 0; n < NS; ++n) sg.copy_to(sa + (unsigned)(sizeof(T) * (n * R::RZ * PL + slot)), job.zf[n] + off);
  };
  // when the planes of level k that its faces and cells read are free: field k+4 into the slot of k-1,
  // flow k+3 into that of k+1 (w on its dual grid: one level up), diff k+2 into that of k-1
  auto stage_next = [&](int k) {
    if (k + 4 <= min(nz, ke + 2)) stage_field(zm, go + 4 * plane);
    if (k + 3 + R::UP <= min(nz, ke + 1 + R::UP)) {
      const long long off = go + (3 + R::UP) * plane;
      const unsigned f = sa + (unsigned)(sizeof(T) * (NS * R::RZ * PL + fo));
      sg.copy_to(f, job.u + off);
      sg.copy_to(f + (unsigned)(sizeof(T) * R::RF * PL), job.v + off);
      sg.copy_to(f + (unsigned)(sizeof(T) * 2 * R::RF * PL), job.w + off);
    }
    if constexpr (DIM < 0)
      if (k + 2 <= ke) sg.copy_to(sa + (unsigned)(sizeof(T) * ((NS * R::RZ + 3 * R::RF) * PL + dm)), job.diff + go + 2 * plane);
  };
  // the slot of level kb-2, which the face below the chunk read, takes level kb+3
  __syncthreads();
  if (kb + 3 <= min(nz, ke + 2)) stage_field(z3, go + 3 * plane);
  T pnext = l_thread && kb + 2 <= min(nz, ke + 1) ? level_const(kb + 2) : (T)0.0;
  for (int k = kb; k <= ke; ++k, lev += plane, go += plane) {
    // level constants of k+2, loaded a level ahead; level k+1 reads them after this level's barrier
    if (l_thread && k + 2 <= min(nz, ke + 1)) rL[((k + 2) & (RL - 1)) * L_N + lane] = pnext;
    if (l_thread && k + 3 <= min(nz, ke + 1)) pnext = level_const(k + 3);
    const long long o = lev + col;
    T fv[NS];
    if constexpr (DIM < 0) {
#pragma unroll
      for (int n = 0; n < NS; ++n) fv[n] = act ? __ldg(job.f[n] + o) : (T)0.0;
    }
    const T* L = rL + (k & (RL - 1)) * L_N;
    const T* Ln = rL + ((k + 1) & (RL - 1)) * L_N;
    T2 *const tVW = reinterpret_cast<T2*>(cur), *const tUR = tVW + CN;
    T2 *const tVWn = reinterpret_cast<T2*>(nxt), *const tURn = tVWn + CN;
    T *const FX = cur + 4 * CN, *const FY = FX + NS * NFX, *const BV = FY + NS * NFY, *const BVn = nxt + (BV - cur);
    if (DIM != 2 || k <= ktop) {
      const int fo2 = R::UP ? ((k + 2) % R::RF) * PL : 0;
      const bool top = k + 1 == nz;
      const T *pu = rU + fo, *pv = rV + fo, *pw = rW + fo;
      const T *pu2 = rU + fo2, *pv2 = rV + fo2, *pw2 = rW + fo2;
      // an x or y face of the cell at plane offset c: along stride st, across stride tr, wsum the w
      // sums and tsum the transverse sums of the two cells, rlo, rhi their reciprocals
      auto h_face = [&](T vel, T cd, T cf, int c, int st, int tr, T wsum, T tsum, T rlo, T rhi, T* out, int ostride) {
        const bool neg = negative(vel);
        const T cmod = fabs(vel) * cd, omc = (T)1.0 - cmod, k6 = r6 * cmod + r6;
        const T r = neg ? rhi : rlo, flux = vel * cf;
        const int oc = c + (neg ? st : 0) + z0, dir = neg ? -st : st;
        const bool wneg = negative(wsum);
        int oz = (wneg ? z1 : zm) - z0;
        T wabs = fabs(wsum);
        if (k == nz) {  // no level above: the difference below, with its sign turned for downward flow
          oz = zm - z0;
          if (wneg) wabs = -wabs;
        }
        const int ot = negative(tsum) ? tr : -tr;
#pragma unroll
        for (int n = 0; n < NS; ++n) {
          const T* p = rF + n * R::RZ * PL + oc;
          const T fc = p[0], fd = p[dir], fu = p[-dir];
          const T a = fc - fu, e = fd - fc;
          T b = omc * ((T)0.5 * e - k6 * (e - a));
          b = b - wabs * (fc - p[oz]) - fabs(tsum) * (fc - p[ot]);
          out[n * ostride] = flux * limit<T>(fc, a, e, b, r);
        }
      };
      // the cell of level k+1 at plane offset c, its w at level k given
      auto next_cell = [&](int c, T wk, T& u, T& v, T& w) {
        u = dual<T, DIM>(pu, pu2, c, top);
        v = dual<T, DIM>(pv, pv2, c, top);
        w = dual<T, DIM>(pw, pw2, c, top);
        return make_cell<T>(cs, Ln[L_WS], Ln[L_CS], u, dual<T, DIM>(pu, pu2, c - 1, top), v,
                            dual<T, DIM>(pv, pv2, c - PW, top), w, wk);
      };
      const T2 ovw = tVW[own], our = tUR[own];
      // the own cell of level k+1, from the staged flow, then the faces of level k
      Cell<T> cn{};
      T un = (T)0.0, vn = (T)0.0, wn = (T)0.0;
      if (k < nz) cn = next_cell(co, w0, un, vn, wn);
      // the tables of level k+1: at once where they have a copy of their own
      auto put_own = [&]() {
        tVWn[own] = T2{cn.vs, cn.ws};
        tURn[own] = T2{cn.us, cn.r};
      };
      Cell<T> bn{};
      T bvn = (T)0.0;
      if (hr >= 0 && k < nz) {
        T bu, bv, bwn;
        bn = next_cell(bco, bw, bu, bv, bwn);
        bvn = hr == 0 ? bv : bu;
        bw = bwn;
      }
      auto put_border = [&]() {
        tVWn[bcell] = T2{bn.vs, bn.ws};
        tURn[bcell] = T2{bn.us, bn.r};
        if (hr == 0) BVn[lane] = bvn;
        if (hc == 0) BVn[TX + lane] = bvn;
      };
      if (DB && k < nz) {
        put_own();
        if (hr >= 0) put_border();
      }
      T fz_hi[NS];
#pragma unroll
      for (int n = 0; n < NS; ++n) fz_hi[n] = (T)0.0;
      if constexpr (DIM == 2) {
        if (k == nz - 1) {
          // the topmost face of w, whose outflow sums take other levels' metrics
          const GF IU{gU, nz}, IV{gV, nz}, IW{gW, nz};
          fz_hi[0] = w0 * tvd_face_z<T, GF, View<T>, Prof<T>, TvdMetricW>(s, prof<T>(s), IU, IV, IW,
                                                                         view<T>(job.zf[0], s), dtm_x2, k, j, i);
        } else {
          z_face(k, w0, zm, z0, z1, z2, ovw.x + cn.vs, our.x + cn.us, our.y, cn.r, L, fz_hi);
        }
      } else if (k < nz) {
        T rhi = cn.r;
        // the downward face below the top level leaves out what flows through the lid
        if (k == nz - 1 && wn != (T)0.0) rhi = make_cell<T>(cs, Ln[L_WS], Ln[L_CS], un, dual<T, DIM>(pu, pu2, co - 1, true), vn,
                                                            dual<T, DIM>(pv, pv2, co - PW, true), (T)0.0, w0).r;
        z_face(k, w0, zm, z0, z1, z2, ovw.x + cn.vs, our.x + cn.us, our.y, rhi, L, fz_hi);
      }
      {
        const T2 nvw = tVW[own + 1];
        h_face(u0, cdx, cx, co, 1, PW, ovw.y + nvw.y, ovw.x + nvw.x, our.y, tUR[own + 1].y, FX + ty * (TX + 1) + tx + 1, NFX);
      }
      {
        const T2 nur = tUR[own + CW];
        h_face(v0, cdy, cy, co, PW, 1, ovw.y + tVW[own + CW].y, our.x + nur.x, our.y, nur.y, FY + (ty + 1) * TX + tx, NFY);
      }
      if (ty == 3) {
        const int o0 = lane + 1;
        const T2 bvw = tVW[o0], bur = tUR[o0], nur = tUR[o0 + CW];
        h_face(BV[lane], cdy, cy, (HY - 1) * PW + lane + Gt::V, PW, 1, bvw.y + tVW[o0 + CW].y, bur.x + nur.x, bur.y, nur.y,
               FY + lane, NFY);
      } else if (ty == 4 && lane < TY) {
        const int o0 = (lane + 1) * CW;
        const T2 bvw = tVW[o0], bur = tUR[o0], nvw = tVW[o0 + 1];
        h_face(BV[TX + lane], cdx, cx, (lane + HY) * PW + Gt::V - 1, 1, PW, bvw.y + nvw.y, bvw.x + nvw.x, bur.y, tUR[o0 + 1].y,
               FX + lane * (TX + 1), NFX);
      }
      // what of the source needs the planes: diffusion, damping, subsidence
      T src[NS], zv[NS];
#pragma unroll
      for (int n = 0; n < NS; ++n) src[n] = (T)0.0;
      auto local_source = [&]() {
        if (job.first && s.th_baroclinic) src[0] = src[0] + ((v0 + (T)s.vgal) * (T)s.mfx - (u0 + (T)s.ugal) * (T)s.mfy);
        if (s.use_vd) {
          // diffusion_point, its level sums of the diffusivity formed once for the NS fields
          const T *pm = rD + dm + co, *p0 = rD + d0 + co;
          const T dmc = pm[0], d0c = p0[0], d2 = d0c + dmc;
          const T kx = (T)s.cx2 * (T)0.25, ky = (T)s.cy2 * (T)0.25;
          const T axm = (d2 + (p0[-1] + pm[-1])) * kx, axp = (d2 + (p0[1] + pm[1])) * kx;
          const T aym = (d2 + (p0[-PW] + pm[-PW])) * ky, ayp = (d2 + (p0[PW] + pm[PW])) * ky;
          const T bm = L[L_CZB] * dmc, bp = L[L_CZA] * d0c;
#pragma unroll
          for (int n = 0; n < NS; ++n) {
            const T* p = rF + n * R::RZ * PL + co;
            const T f0 = p[z0];
            zv[n] = f0;
            T t = axm * (p[z0 - 1] - f0) + axp * (p[z0 + 1] - f0) + aym * (p[z0 - PW] - f0) + ayp * (p[z0 + PW] - f0);
            t = t + bm * (p[zm] - f0);
            if (k < nz) t = t + bp * (p[z1] - f0);
            src[n] = src[n] + t;
          }
        } else {
#pragma unroll
          for (int n = 0; n < NS; ++n) zv[n] = rF[n * R::RZ * PL + co + z0];
        }
        // damping, then forcing's subsidence (the dynamics group's order)
        if (s.damping || s.subs_th || s.subs_q) {
          const Prof<T> P = prof<T>(s);
#pragma unroll
          for (int n = 0; n < NS; ++n) {
            const T* p = rF + n * R::RZ * PL + co;
            const Col3<T> F{p[zm], zv[n], k < nz ? p[z1] : zv[n], k};
            const bool theta = n == 0 && job.first;
            if (s.damping && !(theta && s.passive_th)) src[n] = damping_scalar_point<T>(s, P, k, zv[n], job.row[n], src[n]);
            if (theta ? s.subs_th : s.subs_q)
              src[n] = theta ? subsidence_theta_point<T>(s, P, F, k, j, i, src[n])
                             : subsidence_q_point<T>(s, P, F, job.row[n] - 3, k, j, i, src[n]);
          }
        }
      };
      if constexpr (DB && DIM < 0) local_source();
      if constexpr (DB) asm volatile("cp.async.wait_all;\n" ::: "memory");
      __syncthreads();
      // every face of the level is known
      if constexpr (DB) stage_next(k);
      if (!DB && k < nz) {
        put_own();
        if (hr >= 0) put_border();
      }
#pragma unroll
      for (int n = 0; n < NS; ++n) {
        const T* fx = FX + n * NFX + ty * (TX + 1) + tx;
        const T* fy = FY + n * NFY + ty * TX + tx;
        src[n] = src[n] + (((fx[0] - fx[1]) + (fy[0] - fy[TX])) + (fz_lo[n] * L[L_T1] - fz_hi[n] * L[L_T2]));
        fz_lo[n] = fz_hi[n];
      }
      if constexpr (DIM >= 0) {
        if (act) job.src[o] = src[0];
      } else {
        if constexpr (!DB) local_source();
        if constexpr (CLOUD) {
          // fields 1 and 2 are vapour and liquid
          const CloudProf<T> P{L, k, s};
          simplecloud_point<T>(s, P, k, zv[1], zv[2], zv[0], zv[2], src[0], src[1], src[2]);
        }
#pragma unroll
        for (int n = 0; n < NS; ++n) {
          T zn = zv[n] + dtm_x2 * src[n];
          if ((n > 0 || !job.first) && zn < (T)0.0) zn = (T)0.0;
          if (act) {
            job.out_zf[n][o] = (c1 * fv[n] + c2 * zv[n]) + c2 * zn;
            job.out_f[n][o] = zn;
          }
        }
      }
      u0 = un;
      v0 = vn;
      w0 = wn;
    } else {
      if (act) job.src[o] = (T)0.0;  // w at the top level
    }
    if constexpr (!DB) {
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      __syncthreads();
      stage_next(k);
    }
    // the planes move down a level
    const int zt = zm;
    zm = z0;
    z0 = z1;
    z1 = z2;
    z2 = z3;
    z3 = zt;
    const int dt3 = dm;
    dm = d0;
    d0 = d1;
    d1 = dt3;
    fo = R::UP ? ((k + 2) % R::RF) * PL : PL - fo;
    T* const ct = cur;
    cur = nxt;
    nxt = ct;
  }
}

// The number of chunks the levels are split into.  Where chunks of 8 levels give every resident slot
// a CTA, choose_level_chunks (256 x 256 x 128 in FP64: theta 0.246 ms at its 8 chunks, 0.243 .. 0.268
// for 4 .. 16; momentum 0.247, 0.254 .. 0.265).  On smaller grids, where latency counts, shorter
// chunks: an SM gets m = ceil(tiles n / SMs) CTAs and runs them occ at a time; a CTA takes a level in
// a time that grows with the CTAs beside it, about as 1 + their number (theta, FP64: 1.3 us alone,
// 2.0 us for two), and its first levels cost about two more.  64 x 64 x 65 in FP64: 16 chunks, theta
// 13.7 us (8: 16.2, 22: 18.7, 32: 17.1), subgrid 7.9 (8: 10.4), momentum 12.9 (8: 15.1).
static inline int choose_chunks(int tiles, int occ, int nsm, int levels) {
  if ((long long)tiles * (levels / 8) >= (long long)occ * nsm) return choose_level_chunks(tiles, occ * nsm, levels);
  int best = 1;
  long long best_cost = -1;
  for (int n = 1; n <= 64 && 2 * n <= levels; ++n) {
    const long long m = ((long long)tiles * n + nsm - 1) / nsm, rest = m % occ;
    const long long cost = ((m / occ) * (occ + 1) + (rest ? rest + 1 : 0)) * ((levels + n - 1) / n + 2);
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = n; }
  }
  return best;
}

template <typename T, int NS, bool CLOUD, int DIM>
static int launch(const Scalars& s, const Job<T, NS>& job, cudaStream_t st) {
  const size_t smem = smem_bytes<T, NS, DIM>();
  static LaunchTable table;
  const LaunchLimits lim = launch_limits(table, {(const void*)k_f_tvd<T, NS, CLOUD, DIM>}, NT, smem);
  const int gx = (s.nx + TX - 1) / TX, gy = (s.ny + TY - 1) / TY, levels = s.nz - 1;
  const int nc = s.level_chunks > 0 ? s.level_chunks : choose_chunks(gx * gy, lim.occ, lim.nsm, levels);
  const int kc = (levels + nc - 1) / nc;
  k_f_tvd<T, NS, CLOUD, DIM><<<dim3(gx, gy, (levels + kc - 1) / kc), NT, smem, st>>>(s, job, kc);
  return 1;
}

// flow component DIM: its advective source
template <typename T, int DIM>
static int launch_flow(const Scalars& s, const DevState<T>& d, const T* zf, T* src, cudaStream_t st) {
  Job<T, 1> job{};
  job.u = d.u; job.v = d.v; job.w = d.w;
  job.zf[0] = zf;
  job.src = src;
  return launch<T, 1, false, DIM>(s, job, st);
}

template <typename T>
static int launch_all_flow(const Scalars& s, const DevState<T>& d, cudaStream_t st) {
  return launch_flow<T, 0>(s, d, d.zu, d.su, st) + launch_flow<T, 1>(s, d, d.zv, d.sv, st) +
         launch_flow<T, 2>(s, d, d.zw, d.sw, st);
}

// scalars n0 .. n0+NS-1 (0 is theta, 1 + m the q field m)
template <typename T, int NS, bool CLOUD>
static int launch_scalars(const Scalars& s, const DevState<T>& d, int n0, cudaStream_t st) {
  Job<T, NS> job{};
  job.u = d.u; job.v = d.v; job.w = d.w; job.diff = d.diff;
  for (int n = 0; n < NS; ++n) {
    const int q = n0 + n - 1;
    job.f[n] = q < 0 ? d.th : d.q[q];
    job.zf[n] = q < 0 ? d.zth : d.zq[q];
    job.out_f[n] = q < 0 ? d.th_n : d.q_n[q];
    job.out_zf[n] = q < 0 ? d.zth_n : d.zq_n[q];
    job.row[n] = q < 0 ? 2 : 3 + q;
  }
  job.first = n0 == 0;
  return launch<T, NS, CLOUD, -1>(s, job, st);
}

// theta and every q field: theta, vapour and liquid together under simplecloud (which couples
// them; iqv = 0 and iql = 1 whenever there are two q fields), the rest in groups of up to three
template <typename T>
static int launch_all_scalars(const Scalars& s, const DevState<T>& d, cudaStream_t st) {
  const int ns = 1 + s.nq;
  int n = 0, launches = 0;
  if (s.simplecloud) {
    launches += launch_scalars<T, 3, true>(s, d, 0, st);
    n = 3;
  }
  while (n < ns) {
    const int g = ns - n >= 3 ? 3 : ns - n;
    if (g == 3) launches += launch_scalars<T, 3, false>(s, d, n, st);
    else if (g == 2) launches += launch_scalars<T, 2, false>(s, d, n, st);
    else launches += launch_scalars<T, 1, false>(s, d, n, st);
    n += g;
  }
  return launches;
}

}  // namespace tvdf
}  // namespace KVARIANT
}  // namespace mgpu
