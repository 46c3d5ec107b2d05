// su3.cuh -- SU(3) helpers shared by the force and clover-construction kernels
// (su3.F90, uuu.F90, clover/clover_uuu.F90).
#pragma once
#include "bqcdg_internal.cuh"

namespace bqcdg {

using L64 = Link<double>;
using C64 = cx<double>;

__device__ __forceinline__ void lzero(L64& r) {
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) r.m[a][b] = mkc(0.0, 0.0);
}
// element of u, u^+
__device__ __forceinline__ C64 el(const L64& u, int r, int c, bool dag) {
  return dag ? conjg(u.m[c][r]) : u.m[r][c];
}
// r = op(a) op(b)
__device__ __forceinline__ void mul2(L64& r, const L64& a, bool da, const L64& b, bool db) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      C64 t = el(a, i, 0, da) * el(b, 0, j, db);
      t = t + el(a, i, 1, da) * el(b, 1, j, db);
      t = t + el(a, i, 2, da) * el(b, 2, j, db);
      r.m[i][j] = t;
    }
}
// su3.F90:196-214: p_j += s Im Tr(lambda_j v)
__device__ __forceinline__ void im_tr_j(double p[8], const L64& v, double s) {
  p[0] += s * (v.m[0][1].y + v.m[1][0].y);
  p[1] += s * (v.m[0][1].x - v.m[1][0].x);
  p[2] += s * (v.m[0][0].y - v.m[1][1].y);
  p[3] += s * (v.m[0][2].y + v.m[2][0].y);
  p[4] += s * (v.m[0][2].x - v.m[2][0].x);
  p[5] += s * (v.m[1][2].y + v.m[2][1].y);
  p[6] += s * (v.m[1][2].x - v.m[2][1].x);
  p[7] += s * (v.m[0][0].y + v.m[1][1].y - 2.0 * v.m[2][2].y) * 0.57735026918962573;
}
// su3.F90:216-233: p_j += s Re Tr(lambda_j v)
__device__ __forceinline__ void re_tr_j(double p[8], const L64& v, double s) {
  p[0] += s * (v.m[0][1].x + v.m[1][0].x);
  p[1] += s * (v.m[1][0].y - v.m[0][1].y);
  p[2] += s * (v.m[0][0].x - v.m[1][1].x);
  p[3] += s * (v.m[0][2].x + v.m[2][0].x);
  p[4] += s * (v.m[2][0].y - v.m[0][2].y);
  p[5] += s * (v.m[1][2].x + v.m[2][1].x);
  p[6] += s * (v.m[2][1].y - v.m[1][2].y);
  p[7] += s * (v.m[0][0].x + v.m[1][1].x - 2.0 * v.m[2][2].x) * 0.57735026918962573;
}

__device__ __forceinline__ int site_index(const Geom& g, const int x[4]) {
  return (x[0] >> 1) + g.Lxh * (x[1] + g.L[1] * (x[2] + g.L[2] * x[3]));
}
// coordinates of x shifted by d (+-1) in direction mu, periodic
__device__ __forceinline__ void shift(const Geom& g, const int x[4], int mu, int d, int y[4]) {
#pragma unroll
  for (int k = 0; k < 4; k++) y[k] = x[k];
  y[mu] += d;
  if (y[mu] < 0) y[mu] += g.L[mu];
  if (y[mu] >= g.L[mu]) y[mu] -= g.L[mu];
}
__device__ __forceinline__ int parity_of(const int x[4]) { return (x[0] + x[1] + x[2] + x[3]) & 1; }

__device__ __forceinline__ void load_link(const Geom& g, const double2* gauge, int mu, const int x[4], L64& u) {
  GaugeView<Prec::F64> U{(double2*)gauge, g.stride};
  U.load(mu, parity_of(x), site_index(g, x), u);
}

// staple.F90:28-63: sum over nu != mu of the forward and backward staples.
// With mu a template parameter every shifted coordinate is a register (a
// run-time mu indexes the coordinate arrays, which puts them in local
// memory); staple() dispatches on a run-time mu, uniform across a launch.
template <int MU>
__device__ __forceinline__ void staple_t(const Geom& g, const double2* gauge, const int x[4], L64& st) {
  lzero(st);
#pragma unroll
  for (int nu = 0; nu < 4; nu++) {
    if (nu == MU) continue;
    int x1[4], x2[4], x3[4], x4[4];
    shift(g, x, MU, 1, x1);
    shift(g, x, nu, 1, x2);
    shift(g, x, nu, -1, x3);
    shift(g, x3, MU, 1, x4);
    L64 a, b, c, t, r;
    // uuu_fwd: U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+
    load_link(g, gauge, nu, x1, a);
    load_link(g, gauge, MU, x2, b);
    load_link(g, gauge, nu, x, c);
    mul2(t, a, false, b, true);
    mul2(r, t, false, c, true);
    for (int p = 0; p < 3; p++)
      for (int q = 0; q < 3; q++) st.m[p][q] = st.m[p][q] + r.m[p][q];
    // uuu_bwd: U_nu(x-nu+mu)^+ U_mu(x-nu)^+ U_nu(x-nu)
    load_link(g, gauge, nu, x4, a);
    load_link(g, gauge, MU, x3, b);
    load_link(g, gauge, nu, x3, c);
    mul2(t, a, true, b, true);
    mul2(r, t, false, c, false);
    for (int p = 0; p < 3; p++)
      for (int q = 0; q < 3; q++) st.m[p][q] = st.m[p][q] + r.m[p][q];
  }
}
__device__ __forceinline__ void staple(const Geom& g, const double2* gauge, const int x[4], int mu, L64& st) {
  switch (mu) {
    case 0: staple_t<0>(g, gauge, x, st); break;
    case 1: staple_t<1>(g, gauge, x, st); break;
    case 2: staple_t<2>(g, gauge, x, st); break;
    default: staple_t<3>(g, gauge, x, st); break;
  }
}

// ---------------------------------------------------------------------------
// products with links that stay in memory, for kernels of one thread per link
// ---------------------------------------------------------------------------
// element (r, c) of op(U) of a link in memory (columns of 3)
template <bool DAG>
__device__ __forceinline__ C64 mel(const double2* u, int stride, int r, int c) {
  const double2 t = __ldg(u + (DAG ? r * 3 + c : c * 3 + r) * stride);
  return DAG ? mkc(t.x, -t.y) : mkc(t.x, t.y);
}
__device__ __forceinline__ C64 dmul(double a, C64 b) { return mkc(a * b.x, a * b.y); }
__device__ __forceinline__ C64 dfma(C64 acc, double a, C64 b) { return mkc(fma(a, b.x, acc.x), fma(a, b.y, acc.y)); }

// the row r of op(U) times m is added to (or stored in) t[r][.]; U's row is
// loaded where it is used, so only m and t are live
template <bool DAG, bool ADD>
__device__ __forceinline__ void lmul(L64& t, const double2* u, int stride, const L64& m) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const C64 a0 = mel<DAG>(u, stride, r, 0), a1 = mel<DAG>(u, stride, r, 1), a2 = mel<DAG>(u, stride, r, 2);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      C64 x = ADD ? fma_c(t.m[r][c], a0, m.m[0][c]) : a0 * m.m[0][c];
      x = fma_c(x, a1, m.m[1][c]);
      t.m[r][c] = fma_c(x, a2, m.m[2][c]);
    }
  }
}
// t += m op(U), column by column of op(U)
template <bool DAG>
__device__ __forceinline__ void rmul_add(L64& t, const L64& m, const double2* u, int stride) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const C64 a0 = mel<DAG>(u, stride, 0, c), a1 = mel<DAG>(u, stride, 1, c), a2 = mel<DAG>(u, stride, 2, c);
#pragma unroll
    for (int r = 0; r < 3; r++) {
      C64 x = fma_c(t.m[r][c], m.m[r][0], a0);
      x = fma_c(x, m.m[r][1], a1);
      t.m[r][c] = fma_c(x, m.m[r][2], a2);
    }
  }
}
// m = op(U)
template <bool DAG>
__device__ __forceinline__ void lload(L64& m, const double2* u, int stride) {
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) m.m[r][c] = mel<DAG>(u, stride, r, c);
}

// the same with a run-time dagger
__device__ __forceinline__ C64 mel_rt(const double2* u, int stride, int r, int c, bool dag) {
  const double2 t = __ldg(u + (dag ? r * 3 + c : c * 3 + r) * stride);
  return mkc(t.x, dag ? -t.y : t.y);
}
__device__ __forceinline__ void lload_rt(L64& m, const double2* u, int stride, bool dag) {
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) m.m[r][c] = mel_rt(u, stride, r, c, dag);
}
template <bool ADD>
__device__ __forceinline__ void lmul_rt(L64& t, const double2* u, int stride, bool dag, const L64& m) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const C64 a0 = mel_rt(u, stride, r, 0, dag), a1 = mel_rt(u, stride, r, 1, dag), a2 = mel_rt(u, stride, r, 2, dag);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      C64 x = ADD ? fma_c(t.m[r][c], a0, m.m[0][c]) : a0 * m.m[0][c];
      x = fma_c(x, a1, m.m[1][c]);
      t.m[r][c] = fma_c(x, a2, m.m[2][c]);
    }
  }
}

// the row (y, z, t) shifts by +-1 in a direction (x is shifted by its
// coordinate); shifts in different directions add
struct Shifts {
  int f[4], b[4];    // row shifts, 0 for x
  int xf, xb, xh;    // half coordinates of x + 1, x - 1, x
  int base;
};
__device__ __forceinline__ Shifts make_shifts(const Geom& g, const Site& st) {
  Shifts q;
  int step = g.Lxh;
  q.f[0] = q.b[0] = 0;
#pragma unroll
  for (int d = 1; d < 4; d++) {
    q.f[d] = st.x[d] == g.L[d] - 1 ? -(g.L[d] - 1) * step : step;
    q.b[d] = st.x[d] == 0 ? (g.L[d] - 1) * step : -step;
    step *= g.L[d];
  }
  q.xf = (st.x[0] == g.L[0] - 1 ? 0 : st.x[0] + 1) >> 1;
  q.xb = (st.x[0] == 0 ? g.L[0] - 1 : st.x[0] - 1) >> 1;
  q.xh = st.x[0] >> 1;
  q.base = st.base;
  return q;
}
// entry k, known at run time, without indexing (an indexed array goes to
// local memory)
__device__ __forceinline__ int pick4(int a0, int a1, int a2, int a3, int k) {
  return k < 2 ? (k == 0 ? a0 : a1) : (k == 2 ? a2 : a3);
}
__device__ __forceinline__ int pick(const int a[4], int k) { return pick4(a[0], a[1], a[2], a[3], k); }

}  // namespace bqcdg
