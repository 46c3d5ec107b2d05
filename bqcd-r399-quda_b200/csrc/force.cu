// force.cu -- pseudofermion force kernels for sm_100a (FP64 accumulation).
//
//   hopping part   dsf.F90:75-100 with d/DSFxyzt.F90:77-117, one thread per
//                  link, forward and backward terms of that link fused;
//   clover part    clover_bsa.F90 / clover_ts.F90 build the six sigma_mu_nu
//                  planes w per site, then clover_d.F90:110-264 contracts them
//                  with the clover-leaf staples: one thread per link gathers
//                  the contributions of the three planes through its direction
//                  and of both parities of w, so p is read and written once
//                  per force.
#include "kernels.cuh"
#include "su3.cuh"

namespace bqcdg {

// ---------------------------------------------------------------------------
// hopping force
// ---------------------------------------------------------------------------
// The gamma projections of DSFxyzt.F90:28-60 have two independent spins, the
// half spinor h of project(), and
//   w(ca, cb) = sum_s G_s(ca) conj(b_s(cb)) = sum_k h_k(a)(ca) conj(h_k(b)(cb))
// (twice that for mu = 3, where h keeps two of the spins).  The forward term
// is -s Im Tr(lambda U w_f), the backward one s Im Tr(lambda w_b U^+) =
// -s Im Tr(lambda U w_b^+), so one product U (w_f + w_b^+) serves both.
template <int MU>
__device__ __forceinline__ void dsf_half(const SpinorView<Prec::F64>& v, int i, bool fwd, C64 h[2][3]) {
  if (MU == 3) {
    v.load_pair(i, fwd ? 2 : 0, h);
  } else {
    Spinor<double> p;
    v.load(i, p);
    project<double, false>(p, MU, fwd, h);
  }
}
// w (+)= sum_k a_k conj(b_k)
template <bool ADD>
__device__ __forceinline__ void dsf_outer(L64& w, const C64 a[2][3], const C64 b[2][3]) {
#pragma unroll
  for (int ca = 0; ca < 3; ca++)
#pragma unroll
    for (int cb = 0; cb < 3; cb++) {
      const C64 t = mulc(a[0][ca], b[0][cb]) + mulc(a[1][ca], b[1][cb]);
      w.m[ca][cb] = ADD ? w.m[ca][cb] + t : t;
    }
}
template <int MU>
__device__ __forceinline__ void dsf_planes(L64& w, const SpinorView<Prec::F64>& AF, const SpinorView<Prec::F64>& BH,
                                           const SpinorView<Prec::F64>& AH, const SpinorView<Prec::F64>& BF, int i,
                                           int j) {
  C64 x[2][3], y[2][3];
  dsf_half<MU>(AF, j, true, x);
  dsf_half<MU>(BH, i, true, y);
  dsf_outer<false>(w, x, y);
  dsf_half<MU>(BF, j, false, x);
  dsf_half<MU>(AH, i, false, y);
  dsf_outer<true>(w, x, y);
}

// p(eo,mu,i): link parity eo.  Even links: forward term from (b at i, at at
// x+mu), backward from (a at i, bt at x+mu); odd links swap (a,b)<->(at,bt)
// (dsf.F90:80-98).  A CTA takes the four directions of 32 sites of one
// parity, one warp each, so the site's own spinors come to L1 once.  24^3x48:
// 0.21 ms against 0.42 ms with four spins and two products (252 registers, 2
// CTAs per SM); the spinors, links and momenta it must move take 0.15 ms.
__global__ void __launch_bounds__(kBlock, 3) k_dsf_hop(Geom g, double* p, const double2* gauge, const double2* a,
                                                    const double2* b, const double2* at, const double2* bt,
                                                    double s) {
  const int i = (blockIdx.x >> 1) * 32 + (threadIdx.x & 31);
  const int mu = threadIdx.x >> 5, eo = blockIdx.x & 1, me = mu * 2 + eo, S = g.stride;
  if (i >= g.volh) return;
  const Site st = site_coords(g, i, eo);
  const SpinorView<Prec::F64> BH{(double2*)(eo == 0 ? b : bt), S},  // b-type field here
      AF{(double2*)(eo == 0 ? at : a), S},                          // a-type field at x+mu
      AH{(double2*)(eo == 0 ? a : at), S},                          // a-type field here
      BF{(double2*)(eo == 0 ? bt : b), S};                          // b-type field at x+mu
  L64 w, v;
  switch (mu) {
    case 0: dsf_planes<0>(w, AF, BH, AH, BF, i, neighbour(g, st, i, 0, true)); break;
    case 1: dsf_planes<1>(w, AF, BH, AH, BF, i, neighbour(g, st, i, 1, true)); break;
    case 2: dsf_planes<2>(w, AF, BH, AH, BF, i, neighbour(g, st, i, 2, true)); break;
    default: dsf_planes<3>(w, AF, BH, AH, BF, i, neighbour(g, st, i, 3, true)); break;
  }
  lmul<false, false>(v, gauge + (size_t)(me * 9) * S + i, S, w);
  // the boundary sign of the link (flip_bc), read without indexing
  const int xm = pick4(st.x[0], st.x[1], st.x[2], st.x[3], mu);
  const int bc = pick4(g.bcsign[0], g.bcsign[1], g.bcsign[2], g.bcsign[3], mu);
  const int Lm = pick4(g.L[0], g.L[1], g.L[2], g.L[3], mu);
  const double sgn = bc < 0 && xm == Lm - 1 ? -1.0 : 1.0;
  double q[8];
  double* pp = p + ((size_t)me * g.volh + i) * 8;
#pragma unroll
  for (int k = 0; k < 8; k++) q[k] = pp[k];
  im_tr_j(q, v, (mu == 3 ? -2.0 : -1.0) * s * sgn);
#pragma unroll
  for (int k = 0; k < 8; k++) pp[k] = q[k];
}

void launch_dsf_hop(const Geom& g, double* p, const double2* gauge, const double2* a, const double2* b,
                    const double2* at, const double2* bt, double s, cudaStream_t st) {
  k_dsf_hop<<<(g.volh + 31) / 32 * 2, kBlock, 0, st>>>(g, p, gauge, a, b, at, bt, s);
}

// ---------------------------------------------------------------------------
// sigma_mu_nu planes.  clover_d contracts each plane's w with the clover-leaf
// staples through Re Tr(lambda_j X), and every product X comes with the one in
// which w^+ takes w's place and the rest is reversed; Re Tr(lambda X^+) =
// Re Tr(lambda X), so only H = w + w^+ enters.  The planes hold s H, s the
// force's factor: 9 reals per site instead of 18.
//   field of one parity: [6 planes][9 * stride] doubles, plane order
//   12,13,14,23,24,34 (clover_d.F90:64-71); in a plane double2[4][stride] of
//   (H00, H11), H01, H02, H12, then double[stride] of H22
// ---------------------------------------------------------------------------
struct Herm {
  double d[3];  // diagonal
  C64 o[3];     // H01, H02, H12
};
__device__ __forceinline__ const double* herm_plane(const double* w, int stride, int pl) {
  return w + (size_t)pl * 9 * stride;
}
__device__ __forceinline__ void herm_store(double* w, int stride, int pl, int i, const Herm& h) {
  double* b = w + (size_t)pl * 9 * stride;
  double2* v = reinterpret_cast<double2*>(b);
  v[i] = make_double2(h.d[0], h.d[1]);
#pragma unroll
  for (int k = 0; k < 3; k++) v[(k + 1) * stride + i] = make_double2(h.o[k].x, h.o[k].y);
  b[8 * stride + i] = h.d[2];
}
// sg (+1 or -1) times the plane's matrix at site i
__device__ __forceinline__ void herm_load(const double* b, int stride, int i, double sg, Herm& h) {
  const double2* v = reinterpret_cast<const double2*>(b);
  double2 t = __ldg(v + i);
  h.d[0] = sg * t.x;
  h.d[1] = sg * t.y;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    t = __ldg(v + (k + 1) * stride + i);
    h.o[k] = mkc(sg * t.x, sg * t.y);
  }
  h.d[2] = sg * __ldg(b + 8 * stride + i);
}

// clover_bsa.F90:40-176: w(ca, cb) = sum_s (sigma a)(s, ca) conj(b(s, cb))
__global__ void __launch_bounds__(kBlock) k_clover_bsa(Geom g, double* w, const double2* bf, const double2* af,
                                                       double s) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.volh) return;
  SpinorView<Prec::F64> A{(double2*)af, g.stride}, B{(double2*)bf, g.stride};
  Spinor<double> a, b;
  A.load(i, a);
  B.load(i, b);
#pragma unroll
  for (int pl = 0; pl < 6; pl++) {
    C64 t[3][3];
#pragma unroll
    for (int ca = 0; ca < 3; ca++) {
      C64 q1 = a.c[0][ca], q2 = a.c[1][ca], q3 = a.c[2][ca], q4 = a.c[3][ca];
      C64 g1, g2, g3, g4;
      switch (pl) {
        case 0: g1 = -q1; g2 = q2; g3 = -q3; g4 = q4; break;
        case 1: g1 = -itimes(q2); g2 = itimes(q1); g3 = -itimes(q4); g4 = itimes(q3); break;
        case 2: g1 = q4; g2 = q3; g3 = q2; g4 = q1; break;
        case 3: g1 = -q2; g2 = -q1; g3 = -q4; g4 = -q3; break;
        case 4: g1 = -itimes(q4); g2 = itimes(q3); g3 = -itimes(q2); g4 = itimes(q1); break;
        default: g1 = q3; g2 = -q4; g3 = q1; g4 = -q2;
      }
#pragma unroll
      for (int cb = 0; cb < 3; cb++)
        t[ca][cb] = mulc(g1, b.c[0][cb]) + mulc(g2, b.c[1][cb]) + mulc(g3, b.c[2][cb]) + mulc(g4, b.c[3][cb]);
    }
    Herm h;
#pragma unroll
    for (int c = 0; c < 3; c++) h.d[c] = 2.0 * s * t[c][c].x;
    h.o[0] = s * (t[0][1] + conjg(t[1][0]));
    h.o[1] = s * (t[0][2] + conjg(t[2][0]));
    h.o[2] = s * (t[1][2] + conjg(t[2][1]));
    herm_store(w, g.stride, pl, i, h);
  }
}

void launch_clover_bsa(const Geom& g, double* w, const double2* b, const double2* a, double s, cudaStream_t st) {
  k_clover_bsa<<<nblocks(g.volh), kBlock, 0, st>>>(g, w, b, a, s);
}

// element (r, c) of chiral block chi of the packed A^-1 of site i, read from
// memory: with r, c known at compile time the slot is too, so nothing is
// indexed at run time (a block held in an array and indexed by a loop
// counter went to local memory)
__device__ __forceinline__ C64 ainv_el(const double2* ainv, int stride, int i, int chi, int r, int c) {
  const int slot_up[6][6] = {{-1, 1, 2, 3, 4, 5},    {-1, -1, 6, 7, 8, 9},    {-1, -1, -1, 11, 12, 13},
                             {-1, -1, -1, -1, 14, 15}, {-1, -1, -1, -1, -1, 17}, {-1, -1, -1, -1, -1, -1}};
  if (r == c) {
    const int ds[6] = {0, 0, 10, 10, 16, 16};
    const double2 t = __ldg(ainv + (size_t)(chi * 18 + ds[r]) * stride + i);
    return mkc((r & 1) ? t.y : t.x, 0.0);
  }
  const int slot = r < c ? slot_up[r][c] : slot_up[c][r];
  const double2 t = __ldg(ainv + (size_t)(chi * 18 + slot) * stride + i);
  return r < c ? mkc(t.x, t.y) : conjg(mkc(t.x, t.y));
}

// clover_t_init.F90 + clover_ts.F90: T = (halved) A^-1 in the Dirac basis,
// w planes = Tr_spin(T sigma_mu_nu).  T(s1,c1,s2,c2) = I1 +- I2 with the sign
// + when s1, s2 are both upper or both lower spins.  T is Hermitian, so w is,
// and H = 2 w: the upper triangle in colour is enough.
__global__ void __launch_bounds__(kBlock) k_clover_ts(Geom g, double* w, const double2* ainv, double s) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.volh) return;
  Herm h[6];
#pragma unroll
  for (int c1 = 0; c1 < 3; c1++)
#pragma unroll
    for (int c2 = c1; c2 < 3; c2++) {
      // T(s1,s2) for this colour pair
      C64 T[4][4];
#pragma unroll
      for (int s1 = 0; s1 < 4; s1++)
#pragma unroll
        for (int s2 = 0; s2 < 4; s2++) {
          int k1 = (s1 & 1) * 3 + c1, k2 = (s2 & 1) * 3 + c2;
          C64 e1 = ainv_el(ainv, g.stride, i, 0, k1, k2), e2 = ainv_el(ainv, g.stride, i, 1, k1, k2);
          T[s1][s2] = ((s1 < 2) == (s2 < 2)) ? e1 + e2 : e1 - e2;
        }
      C64 r[6];
      r[0] = -T[0][0] + T[1][1] - T[2][2] + T[3][3];
      r[1] = itimes(T[0][1]) - itimes(T[1][0]) + itimes(T[2][3]) - itimes(T[3][2]);
      r[2] = T[0][3] + T[1][2] + T[2][1] + T[3][0];
      r[3] = -T[0][1] - T[1][0] - T[2][3] - T[3][2];
      r[4] = itimes(T[0][3]) - itimes(T[1][2]) + itimes(T[2][1]) - itimes(T[3][0]);
      r[5] = T[0][2] - T[1][3] + T[2][0] - T[3][1];
#pragma unroll
      for (int pl = 0; pl < 6; pl++) {
        if (c1 == c2) h[pl].d[c1] = 2.0 * s * r[pl].x;
        else h[pl].o[c1 + c2 - 1] = 2.0 * s * r[pl];
      }
    }
#pragma unroll
  for (int pl = 0; pl < 6; pl++) herm_store(w, g.stride, pl, i, h[pl]);
}

void launch_clover_ts(const Geom& g, double* w, const double2* ainv, double s, cudaStream_t st) {
  k_clover_ts<<<nblocks(g.volh), kBlock, 0, st>>>(g, w, ainv, s);
}

// ---------------------------------------------------------------------------
// clover_d (clover_d.F90:110-264)
//
// For the link U_mu(a) and a plane (mu, nu), with the corners d = a + mu, e =
// a + nu, b = d + nu, f = a - nu, c = d - nu and the links u1 = U_nu(d),
// u2 = U_mu(e), u3 = U_nu(a), u4 = U_nu(f), u5 = U_mu(f), u6 = U_nu(c), the
// sixteen products of clover_d_same_eo and clover_d_diff_eo, w folded into
// H = w + w^+ and U_mu(a) taken out, sum to U_mu(a) X with
//   same parity   X = u1 (v^+ Ha + Hb v^+) - u6^+ (v'^+ Ha + Hc v'^+),
//                 v = u3 u2, v' = u4^+ u5
//   other parity  X = (Hd k + k He) u3^+ - (Hd k' + k' Hf) u4,
//                 k = u1 u2^+, k' = u6^+ u5^+
// (times -1 for mu > nu): 8 matrix products per plane and parity in place of
// 20 to 24, and one for the link.  X adds up over the planes, so U_mu(a) is
// applied and Re Tr(lambda_j .) taken once.
// ---------------------------------------------------------------------------
// t (+)= H m
template <bool ADD>
__device__ __forceinline__ void hmul(L64& t, const Herm& h, const L64& m) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    C64 x0 = ADD ? dfma(t.m[0][c], h.d[0], m.m[0][c]) : dmul(h.d[0], m.m[0][c]);
    C64 x1 = ADD ? dfma(t.m[1][c], h.d[1], m.m[1][c]) : dmul(h.d[1], m.m[1][c]);
    C64 x2 = ADD ? dfma(t.m[2][c], h.d[2], m.m[2][c]) : dmul(h.d[2], m.m[2][c]);
    x0 = fma_c(x0, h.o[0], m.m[1][c]);
    x1 = fma_cc(x1, h.o[0], m.m[0][c]);
    x2 = fma_cc(x2, h.o[1], m.m[0][c]);
    t.m[0][c] = fma_c(x0, h.o[1], m.m[2][c]);
    t.m[1][c] = fma_c(x1, h.o[2], m.m[2][c]);
    t.m[2][c] = fma_cc(x2, h.o[2], m.m[1][c]);
  }
}
// t (+)= m H
template <bool ADD>
__device__ __forceinline__ void mulh(L64& t, const L64& m, const Herm& h) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    C64 x0 = ADD ? dfma(t.m[r][0], h.d[0], m.m[r][0]) : dmul(h.d[0], m.m[r][0]);
    C64 x1 = ADD ? dfma(t.m[r][1], h.d[1], m.m[r][1]) : dmul(h.d[1], m.m[r][1]);
    C64 x2 = ADD ? dfma(t.m[r][2], h.d[2], m.m[r][2]) : dmul(h.d[2], m.m[r][2]);
    x0 = fma_cc(x0, h.o[0], m.m[r][1]);
    x1 = fma_c(x1, h.o[0], m.m[r][0]);
    x2 = fma_c(x2, h.o[1], m.m[r][0]);
    t.m[r][0] = fma_cc(x0, h.o[1], m.m[r][2]);
    t.m[r][1] = fma_cc(x1, h.o[2], m.m[r][2]);
    t.m[r][2] = fma_c(x2, h.o[2], m.m[r][1]);
  }
}
__device__ __forceinline__ void adj(L64& m) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    m.m[r][r].y = -m.m[r][r].y;
#pragma unroll
    for (int c = r + 1; c < 3; c++) {
      const C64 t = m.m[r][c];
      m.m[r][c] = conjg(m.m[c][r]);
      m.m[c][r] = conjg(t);
    }
  }
}
// X += the products of every plane through the link with the planes w of the
// link's parity (SAME) or of the other one
template <bool SAME>
__device__ __forceinline__ void clover_d_planes(L64& X, const Shifts& q, const double2* gauge, const double* w, int S,
                                                int i, int mu, int e) {
  const int fmu = pick(q.f, mu), xmu = mu == 0 ? q.xf : q.xh;
  const int id = q.base + fmu + xmu;  // d
#pragma unroll 1
  for (int nu = 0; nu < 4; nu++) {
    if (nu == mu) continue;
    const int lo = mu < nu ? mu : nu, hi = mu < nu ? nu : mu;
    const double* wp = herm_plane(w, S, lo == 0 ? hi - 1 : lo == 1 ? hi + 1 : 5);
    const double sg = mu < nu ? 1.0 : -1.0;
    const int fn = pick(q.f, nu), bn = pick(q.b, nu);
    const int ie = q.base + fn + (nu == 0 ? q.xf : q.xh), jf = q.base + bn + (nu == 0 ? q.xb : q.xh);
    const int ib = q.base + fmu + fn + (nu == 0 ? q.xf : xmu), ic = q.base + fmu + bn + (nu == 0 ? q.xb : xmu);
    const double2 *Um_o = gauge + (size_t)((mu * 2 + 1 - e) * 9) * S, *Un_o = gauge + (size_t)((nu * 2 + 1 - e) * 9) * S,
                  *Un_e = gauge + (size_t)((nu * 2 + e) * 9) * S;
    L64 m, k, t;
    Herm h;
    if (SAME) {
      lload<false>(m, Um_o + ie, S);
      lmul<false, false>(k, Un_e + i, S, m);  // v = u3 u2
      adj(k);
      herm_load(wp, S, i, sg, h);
      mulh<false>(t, k, h);
      herm_load(wp, S, ib, sg, h);
      hmul<true>(t, h, k);
      lmul<false, true>(X, Un_o + id, S, t);  // u1
      lload<false>(m, Um_o + jf, S);
      lmul<true, false>(k, Un_o + jf, S, m);  // v' = u4^+ u5
      adj(k);
      herm_load(wp, S, i, -sg, h);
      mulh<false>(t, k, h);
      herm_load(wp, S, ic, -sg, h);
      hmul<true>(t, h, k);
      lmul<true, true>(X, Un_e + ic, S, t);   // u6^+
    } else {
      lload<true>(m, Um_o + ie, S);
      lmul<false, false>(k, Un_o + id, S, m); // k = u1 u2^+
      herm_load(wp, S, id, sg, h);
      hmul<false>(t, h, k);
      herm_load(wp, S, ie, sg, h);
      mulh<true>(t, k, h);
      rmul_add<true>(X, t, Un_e + i, S);      // u3^+
      lload<true>(m, Um_o + jf, S);
      lmul<true, false>(k, Un_e + ic, S, m);  // k' = u6^+ u5^+
      herm_load(wp, S, id, -sg, h);
      hmul<false>(t, h, k);
      herm_load(wp, S, jf, -sg, h);
      mulh<true>(t, k, h);
      rmul_add<false>(X, t, Un_o + jf, S);    // u4
    }
  }
}

// One thread per link; a CTA takes the four directions of 32 sites of one
// parity, one warp each, so that they share their w planes and most links.
// 24^3x48: 1.30 ms for both parities and 0.73 ms for one, where the 20- to
// 24-product form took 4.92 and 2.46 ms.  (The 8 link classes in sequence over
// the lattice re-read the fields from HBM: 1.24 against 1.02 ms, averaged over
// the two.)  Bound by FP64 arithmetic (per link and both parities 24 products
// with a Hermitian matrix, 90 FMA each, and 25 others, 108 each: 0.68 ms at 18.9
// T FMA/s, FP64 pipe 57 % busy) and by the latency of its gathers, 84 % of which
// L2 serves.  2 CTAs per SM hold X, k, t and a link without spilling; 3 spill 48
// bytes and are no faster.
// eo_w 0, 1: w0 holds the planes of that parity; 2: w0 the even and w1 the
// odd ones, both in one pass over the links
__global__ void __launch_bounds__(kBlock, 2) k_clover_d(Geom g, double* p, const double2* gauge, const double* w0,
                                                        const double* w1, int eo_w) {
  const int i = (blockIdx.x >> 1) * 32 + (threadIdx.x & 31);
  const int me = (threadIdx.x >> 5) * 2 + (blockIdx.x & 1);
  if (i >= g.volh) return;
  const int mu = me >> 1, e = me & 1, S = g.stride;
  const Shifts q = make_shifts(g, site_coords(g, i, e));
  L64 X;
  lzero(X);
  if (eo_w == 2 || eo_w == e) clover_d_planes<true>(X, q, gauge, eo_w == 2 && e ? w1 : w0, S, i, mu, e);
  if (eo_w == 2 || eo_w != e) clover_d_planes<false>(X, q, gauge, eo_w == 2 && !e ? w1 : w0, S, i, mu, e);
  L64 r;
  lmul<false, false>(r, gauge + (size_t)(me * 9) * S + i, S, X);
  double* pp = p + ((size_t)me * g.volh + i) * 8;
  double a[8];
#pragma unroll
  for (int k = 0; k < 8; k++) a[k] = pp[k];
  re_tr_j(a, r, 1.0);
#pragma unroll
  for (int k = 0; k < 8; k++) pp[k] = a[k];
}

void launch_clover_d(const Geom& g, double* p, const double2* gauge, const double* w, int eo_w, cudaStream_t st) {
  const dim3 grid((g.volh + 31) / 32 * 2);
  k_clover_d<<<grid, kBlock, 0, st>>>(g, p, gauge, w, w + clover_w_field(g), eo_w);
}

}  // namespace bqcdg
