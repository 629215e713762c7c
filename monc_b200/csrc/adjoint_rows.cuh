// Scatter of stencil adjoints by rows of a tile.
//
// A point of the momentum adjoint makes 130 contributions to its inputs, one of the subgrid adjoint 51, and
// with one FP64 atomic for each of them the passes ran at the L2's atomic rate.  Here a point first sums what it adds to
// the 3 x 3 x 3 cells around it (Cells), a warp adds up its 32 neighbours in x by shuffles, the tile's HY
// rows add up in y through shared memory, and one atomic per field and level of the stencil is left, plus
// those of the tile's border cells.  At 128 x 128 x 96 the momentum pass went from 305 to 188 us and the
// subgrid pass from 149 to 93; tiles of 4 rows take 215 and 94, the momentum pass split into flow and
// viscosity 85 + 126.  Now bound by the loads' latency at 16 warps an SM (124 registers).
#pragma once

#include "dycore_device.cuh"

namespace mgpu {
namespace hadj {

constexpr int HX = 32, HY = 8;

// contributions of one point to one field; the cells a pass never adds to stay literal zeros and are
// left out by the cell mask of its share and add
struct Cells {
  double a[3][3][3] = {};
  __device__ __forceinline__ void add(int dk, int dj, int di, double v) { a[dk + 1][dj + 1][di + 1] += v; }
};
// mask bit of the cell (dk, dj, di); a mask lists every cell a pass can add to
constexpr unsigned cell(int dk, int dj, int di) { return 1u << (9 * (dk + 1) + 3 * (dj + 1) + di + 1); }
constexpr unsigned xrow(int dk, int dj) { return cell(dk, dj, -1) | cell(dk, dj, 0) | cell(dk, dj, 1); }
constexpr bool has_row(unsigned m, int dk, int dj) { return m & xrow(dk, dj); }
// shared slot of the row (dk, dj != 0) of mask m, counted from 0
constexpr int row_slot(unsigned m, int dk, int dj) {
  int n = 0;
  for (int k = -1; k <= 1; ++k)
    for (int j = -1; j <= 1; j += 2) {
      if (k == dk && j == dj) return n;
      n += has_row(m, k, j);
    }
  return n;
}
constexpr int row_count(unsigned m) { return row_slot(m, 2, 0); }

// this thread's place in its tile.  Threads outside the domain take part with zero contributions
struct Tile {
  Geo g;
  int k, j, i, lane, ty;
  bool in, up;            // the point lies in the domain; level k + 1 exists
  bool first, last, top;  // first, last column and last row of the tile that lie in the domain
  __device__ __forceinline__ explicit Tile(const Scalars& s) : g{s.nx, s.ny, s.nz, s.plane} {
    lane = threadIdx.x;
    ty = threadIdx.y;
    i = blockIdx.x * HX + lane;
    j = blockIdx.y * HY + ty;
    k = blockIdx.z + 1;
    in = i < s.nx && j < s.ny;
    up = k < s.nz;
    first = lane == 0;
    last = (lane == HX - 1 && i < s.nx) || i == s.nx - 1;
    top = ty == HY - 1 || j >= s.ny - 1;
  }
};

template <int NS>
struct Rows {
  double c[NS][HY][HX];
  double e[NS][HY][2];
};
// a row summed in x: the thread's own column and, in the first and last lane, the column beyond it
struct RowSum {
  double c, e;
};

// the rows of mask M summed in x: those with dj = 0 into r (by dk), the others into the shared slots
// from S0 on
template <unsigned M, int S0, int NS>
__device__ __forceinline__ void share_rows(const Cells& x, const Tile& t, Rows<NS>& sh, RowSum (&r)[3]) {
  static_assert(S0 + row_count(M) <= NS, "shared rows");
#pragma unroll
  for (int dk = -1; dk <= 1; ++dk)
#pragma unroll
    for (int dj = -1; dj <= 1; ++dj) {
      if (!has_row(M, dk, dj)) continue;
      const double vm = x.a[dk + 1][dj + 1][0], vp = x.a[dk + 1][dj + 1][2];
      RowSum q{x.a[dk + 1][dj + 1][1], 0.0};
      if (M & cell(dk, dj, 1)) {
        const double up = __shfl_up_sync(0xffffffffu, vp, 1);
        if (!t.first) q.c += up;
        if (t.last) q.e = vp;
      }
      if (M & cell(dk, dj, -1)) {
        const double dn = __shfl_down_sync(0xffffffffu, vm, 1);
        if (!t.last) q.c += dn;
        if (t.first) q.e = vm;  // a first lane is never the last one: the domain's length in x is even
      }
      if (dj == 0) {
        r[dk + 1] = q;
      } else {
        const int n = S0 + row_slot(M, dk, dj);
        sh.c[n][t.ty][t.lane] = q.c;
        if (t.first || t.last) sh.e[n][t.ty][t.first ? 0 : 1] = q.e;
      }
    }
}
// after a barrier: the rows summed in y and added to the adjoint array tg
template <unsigned M, int S0, int NS>
__device__ __forceinline__ void add_rows(double* tg, const Tile& t, const Rows<NS>& sh, const RowSum (&r)[3]) {
  constexpr unsigned EDGE = cell(0, 0, -1) | cell(0, 0, 1) | cell(0, 1, -1) | cell(0, 1, 1) | cell(0, -1, -1) | cell(0, -1, 1);
  if (!t.in) return;
  const int side = t.first ? 0 : 1, ie = t.first ? t.i - 1 : t.i + 1;
#pragma unroll
  for (int dk = -1; dk <= 1; ++dk) {
    const bool lo = has_row(M, dk, -1), mid = has_row(M, dk, 0), hi = has_row(M, dk, 1);
    if (!lo && !mid && !hi) continue;
    if (dk == 1 && !t.up) continue;
    const int nlo = S0 + row_slot(M, dk, -1), nhi = S0 + row_slot(M, dk, 1);
    const bool edge = (t.first || t.last) && (M & (dk < 0 ? EDGE >> 9 : (dk > 0 ? EDGE << 9 : EDGE)));
    double c = mid ? r[dk + 1].c : 0.0, e = mid ? r[dk + 1].e : 0.0;
    if (hi && t.ty > 0) {
      c += sh.c[nhi][t.ty - 1][t.lane];
      if (edge) e += sh.e[nhi][t.ty - 1][side];
    }
    if (lo && !t.top) {
      c += sh.c[nlo][t.ty + 1][t.lane];
      if (edge) e += sh.e[nlo][t.ty + 1][side];
    }
    atomicAdd(tg + t.g.at(t.k + dk, t.j, t.i), c);
    if (edge) atomicAdd(tg + t.g.at(t.k + dk, t.j, ie), e);
    if (lo && t.ty == 0) {
      atomicAdd(tg + t.g.at(t.k + dk, t.j - 1, t.i), sh.c[nlo][0][t.lane]);
      if (edge) atomicAdd(tg + t.g.at(t.k + dk, t.j - 1, ie), sh.e[nlo][0][side]);
    }
    if (hi && t.top) {
      atomicAdd(tg + t.g.at(t.k + dk, t.j + 1, t.i), sh.c[nhi][t.ty][t.lane]);
      if (edge) atomicAdd(tg + t.g.at(t.k + dk, t.j + 1, ie), sh.e[nhi][t.ty][side]);
    }
  }
}

}  // namespace hadj
}  // namespace mgpu
