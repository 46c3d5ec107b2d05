// dslash_split.cu -- the FP64 even/odd clover-Wilson passes of small lattices,
// four threads per site, for sm_100a.
//
// The passes of dslash.cu give a site one thread: a chain of eight hops, each
// a round of loads and about 250 instructions, then the clover blocks.  On a
// lattice that leaves most of the GPU idle that chain is the time of the pass,
// 7 us at 8^4.  Here a CTA of four warps serves 32 sites (lane = site).  Warp
// mu forms the two hops of direction mu, the partial sums meet in shared
// memory, and warp (chi, s) then forms rows 3s..3s+2 of chiral block chi and the
// spin s + 2 chi of the result.  Everything stays in the chiral basis x+- = up
// +- dn, in which the clover blocks and the h terms are diagonal, until the last
// exchange.  So the Wilson and rho terms of a spin, which the one-thread passes
// add to that spin alone, come back from the sum and the difference with its
// partner and carry a rounding of the partner's size.  The z hops, which add the
// neighbours' partners to every spin, bring one like it in either form;
// norm-wise the errors agree (W^+W at 4^4 3.2e-16 and 3.4e-16).
#include "kernels.cuh"
#include "views.cuh"

namespace bqcdg {

constexpr int kSplitSites = 32;

// FP64 fields that the one-thread passes (222 to 248 registers: 2 CTAs of 128
// sites per SM) do in one wave, where the CTAs here, 3 per SM, come to at most
// three per SM for each of theirs: both take a step in time with each CTA more
// on an SM or wave more.  Per FP64 CG iteration with four threads and with one:
//     2048 sites of a parity 21.4 and 40 us, 13824 32.6 and 44.1 (one wave here)
//    17280                   47.3 and 45.1 (two waves, one CTA per SM there)
//    20736                   49.9 and 54.4, 27648 53.5 and 59.0 (two and two)
//    30184                   69.8 and 60.5, 36864 76.3 and 66.8 (three waves)
// and a 24^3x48 solve 179 and 170 ms.
// Four threads per site did nothing for int16 at 10x6x14x18 and slowed the
// FP32 and int16 passes of larger lattices, which wait on issue, not latency.
bool split_sites(Prec p, const Geom& g) {
  constexpr int kSMs = 148;
  const int one = ((g.volh + kBlock - 1) / kBlock + kSMs - 1) / kSMs;
  const int four = ((g.volh + kSplitSites - 1) / kSplitSites + kSMs - 1) / kSMs;
  return p == Prec::F64 && !g.clover_t && one <= 2 && four <= 3 * one;
}
int site_blocks(Prec p, const Geom& g) {
  return split_sites(p, g) ? (g.volh + kSplitSites - 1) / kSplitSites : nblocks(g.volh);
}

// rows 3S..3S+2 of a packed Hermitian block times x (clover_block_mv)
template <int S>
__device__ __forceinline__ void rows_mv(const cx<double> a[18], const cx<double> x[6], cx<double> y[3]) {
  constexpr int up[6][6] = {{0, 1, 2, 3, 4, 5},    {-1, 0, 6, 7, 8, 9},    {-1, -1, 10, 11, 12, 13},
                            {-1, -1, -1, 10, 14, 15}, {-1, -1, -1, -1, 16, 17}, {-1, -1, -1, -1, -1, 16}};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int r = 3 * S + k;
    cx<double> t = ((r & 1) ? a[up[r][r]].y : a[up[r][r]].x) * x[r];
#pragma unroll
    for (int c = 0; c < 6; c++) {
      if (c < r) t = fma_cc(t, a[up[c][r]], x[c]);
      if (c > r) t = fma_c(t, a[up[r][c]], x[c]);
    }
    y[k] = t;
  }
}
__device__ __forceinline__ void rows_mv(int s, const cx<double> a[18], const cx<double> x[6], cx<double> y[3]) {
  if (s == 0) rows_mv<0>(a, x, y);
  else rows_mv<1>(a, x, y);
}

// the slots of block chi of site i that rows 3s..3s+2 need
__device__ __forceinline__ void load_rows(const CloverView<Prec::F64>& A, int i, int chi, int s, cx<double> a[18]) {
  const double2* v = A.v + (size_t)(chi * 18) * A.stride + i;
#pragma unroll
  for (int k = 0; k < 18; k++) {
    const bool upper = k <= 13, lower = !(k <= 2 || k == 6);
    if (s == 0 ? upper : lower) {
      const double2 t = __ldg(v + k * A.stride);
      a[k] = mkc(t.x, t.y);
    }
  }
}

enum class Pass { First, Second, SecondSum, Cg };

// Pass::First: out = Ainv_oo D_oe t, (1 -+ i h g5) out      (k_pass1)
// Pass::Second: out = A_ee x + bcoef D_eo t + rho x (+ h term), SecondSum
//   with the |out|^2 block partials                           (k_pass2)
// Pass::Cg: r -= alpha (the same), |r|^2 block partials       (k_cg_pass4)
// (3 CTAs per SM: at 4 the 128 registers spill, 4.03 against 4.13 ms for the
// 8^4 solve)
template <bool DAG, Pass W>
__global__ void __launch_bounds__(128, 3)
    k_split(Geom g, SpinorPtr outp, SpinorPtr tp, SpinorPtr xp, const void* gauge, CloverPtr ap, int has_clover,
            double bcoef, double hval, double rho, RedScratch red, const CgScalars* cg, AlphaFin fin) {
  using R = double;
  using R2 = double2;
  constexpr Prec P = Prec::F64;
  constexpr int e = W == Pass::First ? 1 : 0;  // parity of the output sites
  __shared__ R2 part[4][12][kSplitSites];  // [direction][chi * 6 + spin * 3 + colour][site]
  __shared__ R2 z4[4][3][kSplitSites];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chi = warp >> 1, s = warp & 1;
  const int extra = fin.partial ? 1 : 0;
  const int sb = (int)blockIdx.x - extra, nsb = (int)gridDim.x - extra;
  if (sb < 0) {
    // alpha of the second pass before (k_pass1's extra CTA)
    chain_wait();
    double tot[1];
    final_sum<1>(after_wait(fin.partial), fin.stride, nsb, tot);
    if (threadIdx.x == 0 && !fin.cg->done) cg_set_alpha(fin.cg, tot[0]);
    return;
  }
  if (retired(cg)) return;
  // threads beyond the last site work on it too, and store nothing
  const int i0 = sb * kSplitSites + lane;
  const bool live = i0 < g.volh;
  const int i = live ? i0 : g.volh - 1;
  const auto U = gview<P>(gauge, g);
  const Site st = site_coords(g, i, e);

  chain_wait();
  const bool stopped = cg && cg->done;
  const auto t = after_wait(sview<P>(tp, g.stride));
  Spinor<R> b;
  zero(b);
  const R hs = W == Pass::First ? 1.0 : bcoef;
  if (warp == 0) wilson_hop_mu<P, DAG>(g, e, i, st, t, U, b, hs, 0);
  else if (warp == 1) wilson_hop_mu<P, DAG>(g, e, i, st, t, U, b, hs, 1);
  else if (warp == 2) wilson_hop_mu<P, DAG>(g, e, i, st, t, U, b, hs, 2);
  else wilson_hop_mu<P, DAG>(g, e, i, st, t, U, b, hs, 3);
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const cx<R> u = b.c[k / 3][k % 3], d = b.c[k / 3 + 2][k % 3];
    part[warp][k][lane] = make_double2(u.x + d.x, u.y + d.y);
    part[warp][6 + k][lane] = make_double2(u.x - d.x, u.y - d.y);
  }
  cx<R> a[18], z[3];  // rows of A_ee or A_oo^-1
  if (has_clover) load_rows(cview<P>(ap, g.stride), i, chi, s, a);
#pragma unroll
  for (int c = 0; c < 3; c++) z[c] = mkc<R>(0, 0);
  if constexpr (W != Pass::First) {
    // the site-local terms: rows of A_ee x and of rho x
    Spinor<R> x;
    after_wait(sview<P>(xp, g.stride)).load(i, x);
    cx<R> xc[6];
#pragma unroll
    for (int k = 0; k < 6; k++)
      xc[k] = chi == 0 ? x.c[k / 3][k % 3] + x.c[k / 3 + 2][k % 3] : x.c[k / 3][k % 3] - x.c[k / 3 + 2][k % 3];
    // x itself is half the sum (difference) of its chiral parts
    const R own = 0.5 * (rho + (has_clover ? 0.0 : 1.0));
    if (has_clover) rows_mv(s, a, xc, z);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const cx<R> xo = s == 0 ? xc[c] : xc[3 + c];
      z[c] = z[c] + own * xo;
      if (!has_clover && hval != 0.0) z[c] = z[c] + (chi == 0 ? 0.5 : -0.5) * hval * itimes(xo);
    }
  }
  if (stopped) return;
  __syncthreads();
  if (W == Pass::First && has_clover) {
    // every row needs the whole chiral vector
    cx<R> xc[6];
#pragma unroll
    for (int k = 0; k < 6; k++) {
      xc[k] = mkc<R>(0, 0);
#pragma unroll
      for (int m = 3; m >= 0; m--) {
        const R2 v = part[m][chi * 6 + k][lane];
        xc[k] = xc[k] + mkc<R>(v.x, v.y);
      }
    }
    rows_mv(s, a, xc, z);
  } else {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      cx<R> h = mkc<R>(0, 0);
#pragma unroll
      for (int m = 3; m >= 0; m--) {
        const R2 v = part[m][warp * 3 + c][lane];
        h = h + mkc<R>(v.x, v.y);
      }
      z[c] = z[c] + 0.5 * h;
    }
  }
  if (W == Pass::First && hval != 0.0) {
    // (1 + i h g5) is 1 +- i h on the chiral parts
#pragma unroll
    for (int c = 0; c < 3; c++) z[c] = z[c] + (chi == 0 ? hval : -hval) * itimes(z[c]);
  }
#pragma unroll
  for (int c = 0; c < 3; c++) z4[warp][c][lane] = make_double2(z[c].x, z[c].y);
  __syncthreads();
  // spin s + 2 chi of the result: up = z+ + z-, dn = z+ - z-
  cx<R> o[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const R2 v = z4[warp ^ 2][c][lane];
    o[c] = chi == 0 ? mkc<R>(z[c].x + v.x, z[c].y + v.y) : mkc<R>(v.x - z[c].x, v.y - z[c].y);
  }
  const int sp = s + 2 * chi;
  double acc[1] = {0.0};
  const auto out = after_wait(sview<P>(outp, g.stride));
  if (W == Pass::Cg) {
    const R al = cg->alpha;  // set by the launch before
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double2 r = ld_field(out.v + (c * 4 + sp) * out.stride + i);
      o[c] = mkc(r.x, r.y) - al * o[c];
    }
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    if (live) out.v[(c * 4 + sp) * out.stride + i] = make_double2(o[c].x, o[c].y);
    acc[0] += norm2(o[c]);
  }
  if (W == Pass::SecondSum || W == Pass::Cg) {
    if (!live) acc[0] = 0.0;
    block_reduce_store<1>(acc, red.partial, red.maxblocks, sb);
  }
}

void launch_split_pass1(const Geom& g, bool dag, SpinorPtr out, SpinorPtr in, const void* gauge, CloverPtr a,
                        const OpParams& op, const CgScalars* cg, cudaStream_t s, AlphaFin fin, bool chain) {
  const dim3 grid(site_blocks(Prec::F64, g) + (fin.partial ? 1 : 0));
  const int hc = op.csw_kappa != 0.0;
  const double hv = dag ? op.h : -op.h;
#define SP1(D)                                                                                              \
  launch_chain(chain, k_split<D, Pass::First>, grid, 128, s, g, out, in, SpinorPtr{}, gauge, a, hc, 0.0, hv, 0.0, \
               RedScratch{}, cg, fin)
  if (dag) SP1(true); else SP1(false);
#undef SP1
}

void launch_split_pass2(const Geom& g, bool dag, SpinorPtr out, SpinorPtr t, SpinorPtr x, const void* gauge,
                        CloverPtr a, const OpParams& op, RedScratch red, const CgScalars* cg, cudaStream_t s,
                        bool chain) {
  const dim3 grid(site_blocks(Prec::F64, g));
  const int hc = op.csw_kappa != 0.0;
  const double bcoef = -op.kappa * op.kappa / (1.0 + op.h * op.h), hv = dag ? -op.h : op.h;
#define SP2(D, W)                                                                                                   \
  launch_chain(chain, k_split<D, W>, grid, 128, s, g, out, t, x, gauge, a, hc, bcoef, hv, op.rho, red, cg, AlphaFin{})
  if (cg) SP2(false, Pass::SecondSum);
  else if (dag) SP2(true, Pass::Second);
  else SP2(false, Pass::Second);
#undef SP2
}

void launch_split_pass4(const Geom& g, SpinorPtr t, SpinorPtr q, const void* gauge, CloverPtr a, const OpParams& op,
                        SpinorPtr r, RedScratch red, const CgScalars* cg, cudaStream_t s) {
  const double bcoef = -op.kappa * op.kappa / (1.0 + op.h * op.h);
  launch_chain(true, k_split<true, Pass::Cg>, dim3(site_blocks(Prec::F64, g)), 128, s, g, r, t, q, gauge, a,
               (int)(op.csw_kappa != 0.0), bcoef, -op.h, op.rho, red, cg, AlphaFin{});
}

}  // namespace bqcdg
