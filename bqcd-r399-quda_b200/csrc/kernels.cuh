// kernels.cuh -- host-side declarations of the sm_100a kernels (launchers).
#pragma once

#include <cuda_runtime.h>
#include "bqcdg_internal.cuh"

namespace bqcdg {

// type-erased device pointers handed from the runtime to the launchers
struct SpinorPtr {
  void* v = nullptr;
  float* norm = nullptr;  // F16 only
  long long rsb = 0;      // bytes from one RHS's field to the next (batched launches)
  long long rsnb = 0;     // same for the norms
};

// the field of right-hand side r in a batched SpinorPtr
__host__ __device__ __forceinline__ SpinorPtr rhs_of(SpinorPtr p, int r) {
  SpinorPtr q = p;
  if (r) {
    q.v = (char*)p.v + r * p.rsb;
    if (p.norm) q.norm = (float*)((char*)p.norm + r * p.rsnb);
  }
  return q;
}
struct CloverPtr {
  void* v = nullptr;
  float* norm = nullptr;  // F16 only
};

// reduction scratch: per-block partials + arrival counter
struct RedScratch {
  double* partial = nullptr;  // [nval][maxblocks]
  unsigned int* counter = nullptr;
  int maxblocks = 0;
};

// scalars of a CG kept in device memory (no host round trip per iteration)
struct CgScalars {
  double rtr;       // |r|^2 after the latest update
  double rtr_old;   // |r|^2 of the previous iteration
  double beta;
  double stop_rtr;  // converged when rtr <= stop_rtr
  double delta2;    // sloppy solver: reliable update when rtr < delta2 * maxr2 (0: never)
  double maxr2;     // largest |r|^2 since the last reliable update
  int iter;         // iterations completed
  int maxiter;
  int done;         // 0 running, 1 converged, 2 reliable update requested, 3 maxiter, 4 NaN
  int last_ru;      // iteration of the last reliable update
  int ru_every;     // also update after this many iterations without one (0: never)
  double paap;      // p.(A p) = |M p|^2
  double alpha;
  int live;         // the iteration that alpha belongs to (iter + 1 when it was set)
};

struct OpParams {
  double kappa;
  double csw_kappa;
  double h;
  double rho;
};

// A launch that may start while the kernel before it in the stream drains
// (programmatic stream serialization), when chain is set.  Only for kernels
// whose threads all call chain_wait (bqcdg_internal.cuh, which has the rules),
// and only where no launch chained before it writes the links, the clover
// fields or whatever else the kernel reads before chain_wait.  Without it
// about 2.2 us pass between two launches; with it the next kernel's CTAs are
// resident by then, with their index arithmetic done and, in the int16 passes,
// their links on their way.  Mixed solves: 19.1 -> 13.5 ms at 16^3x32, 10.6 ->
// 7.1 ms at 10x6x14x18, 248 -> 244 ms at 32^3x64; FP64 CG: 5.7 -> 4.0 ms at
// 8^4, 175 -> 172 ms at 24^3x48; FP32: Wilson at 12x20x28x36 8.4 -> 6.7 ms, 12
// systems at 12^3x24 48.3 -> 43.2 ms.
template <typename... KP, typename... A>
inline void launch_chain(bool chain, void (*k)(KP...), dim3 grid, int block, cudaStream_t s, A... a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = chain ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, KP(a)...);  // an error is seen by the caller's cudaGetLastError
}

// the iteration a k_cg_pupdate launch belongs to, per right-hand side
struct CgExpect {
  int n[kMaxRhs];
};

constexpr int kBlock = 128;
inline int nblocks(int n) { return (n + kBlock - 1) / kBlock; }

// ---- stencil and clover operators (dslash.cu) ----
void launch_dslash(Prec p, const Geom& g, int e, bool dag, SpinorPtr out, SpinorPtr in, const void* gauge,
                   cudaStream_t s);
// out = A in (mult_a); in-place allowed (mult_ao)
void launch_clover_mult(Prec p, const Geom& g, SpinorPtr out, SpinorPtr in, CloverPtr a, cudaStream_t s);
// in-place LDL solve with the B factors (F64 only)
void launch_clover_mult_b(const Geom& g, double2* x, const double2* b, cudaStream_t s);

// The passes of an operator or a CG iteration.  nr > 1 (FP32 and int16): nr
// right-hand sides in one launch, fields at SpinorPtr::rsb strides, cg an array
// of nr entries; a retired one returns at once.  g.clover_t: the clover fields
// hold T and each pass forms A(kappa) and A(kappa)^-1 per site, at op.kappa or
// at kappa_rhs[k] for right-hand side k, which also sets its hopping
// coefficient.  rho_rhs: one shift per right-hand side (device), in place of
// op.rho in the second passes.
//
// The |M~ p|^2 block partials that a second pass with cg left in red.partial
// (slot 0 of each RHS).  The k_pass1 launch after it, given this, sums them in
// one more CTA per RHS (final_sum) and sets that RHS's paap and alpha = rtr /
// paap, so no CTA of the second pass waits for an arrival counter.
struct AlphaFin {
  const double* partial = nullptr;
  int stride = 0;  // RedScratch::maxblocks
  CgScalars* cg = nullptr;
};
// first half of mtil / mtil_dag: out_o = [(1 -+ i h g5)] Ainv_oo D_oe in_e
void launch_mtil_pass1(Prec p, const Geom& g, bool dag, SpinorPtr out_o, SpinorPtr in_e, const void* gauge,
                       CloverPtr ainv_oo, const OpParams& op, const CgScalars* cg, cudaStream_t s, int nr = 1,
                       const double* kappa_rhs = nullptr, AlphaFin fin = AlphaFin{}, bool chain = false);
// second half: out_e = A_ee in_e + b D_eo t_o (+ h term for Wilson) + rho in_e;
// with cg (dag = false only) also the |out|^2 block partials
void launch_mtil_pass2(Prec p, const Geom& g, bool dag, SpinorPtr out_e, SpinorPtr t_o, SpinorPtr in_e,
                       const void* gauge, CloverPtr a_ee, const OpParams& op, RedScratch red, const CgScalars* cg,
                       cudaStream_t s, int nr = 1, const double* rho_rhs = nullptr, const double* kappa_rhs = nullptr,
                       bool chain = false);
// CG-fused second half of mtil_dag: Ap = A_ee q + b D_eo t_o + rho q computed in
// registers; r -= alpha Ap and the |r|^2 block partials (x += alpha p follows in
// k_cg_pupdate).  Precision P for the stencil fields, r in XP (F64 for the FP64
// solver, F32 for the sloppy one)
void launch_cg_pass4(Prec p, const Geom& g, SpinorPtr t_o, SpinorPtr q_e, const void* gauge, CloverPtr a_ee,
                     const OpParams& op, SpinorPtr r, RedScratch red, const CgScalars* cg, cudaStream_t s, int nr = 1,
                     const double* rho_rhs = nullptr, const double* kappa_rhs = nullptr);
// queued after it: sums the |r|^2 partials (one CTA per right-hand side, the
// fixed-order final_sum) and takes the CG scalar step (cg_scalar_step: beta, the
// stop tests).  nsb: site blocks per RHS of that k_cg_pass4 launch.
void launch_cg_step(RedScratch red, CgScalars* cg, int nr, int nsb, cudaStream_t s);
// register-blocked batched passes (dslash_multi.cu): one thread serves one
// site of nbt (2 or 4) right-hand sides, so each link and clover block is
// loaded and decoded once for all of them.  Sloppy precisions (F32, F16)
// and h = 0 only; pass 2 is the non-dagger one with its block partials (cg
// required there and in pass 4).
void launch_mtil_pass1_n(Prec p, const Geom& g, bool dag, SpinorPtr out_o, SpinorPtr in_e, const void* gauge,
                         CloverPtr ainv_oo, const OpParams& op, const CgScalars* cg, cudaStream_t s, int nr,
                         int nbt, AlphaFin fin = AlphaFin{}, bool chain = false);
void launch_mtil_pass2_n(Prec p, const Geom& g, SpinorPtr out_e, SpinorPtr t_o, SpinorPtr in_e, const void* gauge,
                         CloverPtr a_ee, const OpParams& op, RedScratch red, const CgScalars* cg, cudaStream_t s,
                         int nr, const double* rho_rhs, int nbt);
void launch_cg_pass4_n(Prec p, const Geom& g, SpinorPtr t_o, SpinorPtr q_e, const void* gauge, CloverPtr a_ee,
                       const OpParams& op, SpinorPtr r, RedScratch red, const CgScalars* cg, cudaStream_t s, int nr,
                       const double* rho_rhs, int nbt);
// the same three passes of FP64 fields with four threads per site
// (dslash_split.cu), which the launchers above take where split_sites says so:
// one right-hand side, stored clover blocks.  site_blocks: the block partials
// of a pass, at most kRedVals maxblocks
bool split_sites(Prec p, const Geom& g);
int site_blocks(Prec p, const Geom& g);
void launch_split_pass1(const Geom& g, bool dag, SpinorPtr out, SpinorPtr in, const void* gauge, CloverPtr a,
                        const OpParams& op, const CgScalars* cg, cudaStream_t s, AlphaFin fin, bool chain);
void launch_split_pass2(const Geom& g, bool dag, SpinorPtr out, SpinorPtr t, SpinorPtr x, const void* gauge,
                        CloverPtr a, const OpParams& op, RedScratch red, const CgScalars* cg, cudaStream_t s,
                        bool chain);
void launch_split_pass4(const Geom& g, SpinorPtr t, SpinorPtr q, const void* gauge, CloverPtr a, const OpParams& op,
                        SpinorPtr r, RedScratch red, const CgScalars* cg, cudaStream_t s);
// p = r + beta p, and the x += alpha p of iteration expect.n[rhs] if that
// iteration ran
void launch_cg_pupdate(Prec p, const Geom& g, SpinorPtr pvec, SpinorPtr r, CgScalars* cg, cudaStream_t s,
                       int nr, SpinorPtr x, const CgExpect& expect, bool chain = false);

// both, for one right-hand side: every CTA sums the partials itself.  The
// stepped scalars go to `next`; when the iteration did not run they are those
// of `cur`.  One launch less, at one more reading of all partials per CTA.  Per
// iteration, apart and together: FP64 24.6 and 21.4 us at 64 partials (8^4),
// 32.2 and 30.5 at 256, FP32 57 and 54 at 256, int16 37.9 and 34.5 at 60
// (10x6x14x18), 40.3 and 37.1 at 215, 43.4 and 43.4 at 224, but 41.4 and 44.3
// at 236 and 43.5 and 48.8 at 256; from 384 on FP32 loses as well.
inline bool fused_step(Prec p, int nsb) { return nsb <= (p == Prec::F16 ? 216 : 256); }
void launch_cg_update(Prec p, const Geom& g, SpinorPtr pvec, SpinorPtr r, SpinorPtr x, const CgScalars* cur,
                      CgScalars* next, RedScratch red, int nsb, cudaStream_t s);

// ---- block solver (blockcg.cu) ----
// out[i * s + j] = <a_i, b_j> (FP64) for two blocks of s <= 16 FP32 fields
// (batched layout); partial: block_gram_scratch_pairs() complex doubles
int block_gram_scratch_pairs();
void launch_block_gram(const Geom& g, int s, SpinorPtr a, SpinorPtr b, double2* partial, double2* out,
                       cudaStream_t st);
// out_j = sum_k in1_k m1[k * s + j] (+ sum_k in2_k m2[k * s + j] when in2.v):
// right multiplication of FP32 blocks by s x s complex matrices; out may be
// in1 or in2
void launch_block_combine(const Geom& g, int s, SpinorPtr out, SpinorPtr in1, const float2* m1, SpinorPtr in2,
                          const float2* m2, cudaStream_t st);

// ---- configuration files (confio.cu) ----
// time slice t of the resident FP64 links in the order and byte order of
// BQCD's slice files (24 big-endian complex per site, 384 bytes), and back
// with the third column rebuilt; *acc ^= the raw CRC register of the slice
// (zero it first; cksum's length and complement are applied on the host)
cudaError_t launch_links_to_file(const Geom& g, const double2* gauge, int t, void* out, unsigned* acc,
                                 cudaStream_t s);
cudaError_t launch_links_from_file(const Geom& g, const void* in, int t, double2* gauge, unsigned* acc,
                                   cudaStream_t s);

// ---- BLAS / conversions (blas.cu) ----
// r = b - Ax (F64), copy r into p (precision pp); res2[0] = |r|^2, res2[1] = |b|^2
void launch_residual(const Geom& g, double2* r, const double2* b, const double2* ax, Prec pp, SpinorPtr p,
                     RedScratch red, double* res2, cudaStream_t s);
// reliable-update helpers: *out = <r32, p> (real), then p = r + beta (p - rpc r)
void launch_rdot(const Geom& g, SpinorPtr r32, Prec pp, SpinorPtr p, RedScratch red, double* out, cudaStream_t s);
// r = b - Ax in FP32, res3 = {|r|^2, |b|^2, <r, p>} for a sloppy direction p
void launch_update_residual(const Geom& g, SpinorPtr r32, const double2* b, const double2* ax, Prec pp, SpinorPtr p,
                            RedScratch red, double* res3, cudaStream_t s);
void launch_p_reorth(const Geom& g, Prec pp, SpinorPtr p, SpinorPtr r32, double rpc, double beta, cudaStream_t s);
// x = (1 + i h gamma_5) x (h_mult_b, h_mult.F90:51-82), F64
void launch_h_mult_b(const Geom& g, double2* x, double h, cudaStream_t s);
// halved inverse blocks from the LDL factors B (6 unit solves per block)
void launch_ainv_from_b(const Geom& g, double2* ainv, const double2* b, cudaStream_t s);
// generic copy/convert between spinor precisions
void launch_spinor_convert(const Geom& g, Prec pout, SpinorPtr out, Prec pin, SpinorPtr in, cudaStream_t s);
// x64 += xs (F32), xs = 0
void launch_accum_x(const Geom& g, double2* x, float4* xs, cudaStream_t s);
// |v|^2 of an F64 spinor -> *out (device)
void launch_norm2(const Geom& g, const double2* v, RedScratch red, double* out, cudaStream_t s);
// dot <a,b> real part of F64 spinors -> *out
void launch_dot(const Geom& g, const double2* a, const double2* b, RedScratch red, double* out, cudaStream_t s);
// y = a*x + y (F64)
void launch_axpy(const Geom& g, double a, const double2* x, double2* y, cudaStream_t s);
void launch_zero(const Geom& g, Prec p, SpinorPtr v, cudaStream_t s);

// ---- layout conversions (convert.cu) ----
// Fortran SPINCOL_FIELD complex(4,3,volh) <-> device F64 spinor
void launch_spinor_from_fortran(const Geom& g, double2* dev, const double2* host_layout, cudaStream_t s);
void launch_spinor_to_fortran(const Geom& g, double2* host_layout, const double2* dev, cudaStream_t s);
// Fortran GAUGE_FIELD complex(3,3,volh,0:1,4) -> device F64 links (periodic);
// flipped != 0: the input carries flip_bc's boundary sign, which is removed
void launch_gauge_from_fortran(const Geom& g, double2* dev, const double2* host_layout, int flipped, cudaStream_t s);
void launch_gauge_to_fortran(const Geom& g, double2* host_layout, const double2* dev, int flipped, cudaStream_t s);
// Fortran CLOVER_FIELD_A/B (18,2,volh) for one parity -> device F64 [36][stride]
void launch_clover_from_fortran(const Geom& g, double2* dev, const double2* host_layout, cudaStream_t s);
void launch_clover_to_fortran(const Geom& g, double2* host_layout, const double2* dev, cudaStream_t s);
// sloppy copies
void launch_gauge_demote(const Geom& g, Prec p, void* out, const double2* in, cudaStream_t s);
void launch_clover_demote(const Geom& g, Prec p, CloverPtr out, const double2* in, cudaStream_t s);
// gauge-field SU(3) check: max |U U^+ - 1| and max |det U - 1| -> out[2]
void launch_gauge_check(const Geom& g, const double2* gauge, RedScratch red, double* out, cudaStream_t s);

// ---- forces (force.cu) ----
// hopping force (dsf.F90:75-100): p(eo,mu) from a,b (even) and at,bt (odd)
void launch_dsf_hop(const Geom& g, double* p, const double2* gauge, const double2* a, const double2* b,
                    const double2* at, const double2* bt, double s, cudaStream_t st);
// The sigma_mu_nu planes w of one parity as s (w + w^+), 9 reals per plane and
// site (force.cu): clover_w_field(g) doubles per parity
inline size_t clover_w_field(const Geom& g) { return (size_t)54 * g.stride; }
// of clover_bsa, from the spinors b, a of that parity
void launch_clover_bsa(const Geom& g, double* w, const double2* b, const double2* a, double s, cudaStream_t st);
// of clover_ts, from the halved inverse blocks (clover_t_init + ts)
void launch_clover_ts(const Geom& g, double* w, const double2* ainv, double s, cudaStream_t st);
// clover_d: p(link) += contributions of the planes w of parity eo_w, or, with
// eo_w = 2, of both parities (w the even field, the odd one after it) in one
// pass over the links
void launch_clover_d(const Geom& g, double* p, const double2* gauge, const double* w, int eo_w, cudaStream_t st);

// ---- clover construction (clover_init.cu) ----
// clover_init.F90 + clover_inv.F90 on device: A, Ainv, B of each parity whose
// pointers are given (null: not computed), in chunks of clover_init_chunk(g)
// sites through tmp (clover_init_tmp(g) complex: the six field strengths of a
// chunk, 5 complex each)
int clover_init_chunk(const Geom& g);
inline size_t clover_init_tmp(const Geom& g) { return (size_t)30 * clover_init_chunk(g); }
void launch_clover_init(const Geom& g, const double2* gauge, double csw_kappa, double2* a[2], double2* ainv[2],
                        double2* b[2], double2* tmp, cudaStream_t s);
// T = (-c_sw / 8)(p +- q) of each chiral block, packed like A, for the
// parities whose pointer is given: the kappa-independent part of the clover
// term, A(kappa) = 1 + kappa T (clover_init.F90:46-77, clover_init3)
void launch_clover_t(const Geom& g, const double2* gauge, double csw, double2* t[2], double2* tmp, cudaStream_t s);
// 2 sum log det over the halved 1/D of B (clover_action.F90)
void launch_clover_action(const Geom& g, const double2* b, RedScratch red, double* out, cudaStream_t s);

// ---- seeded synthetic inputs (gauge_gen.cu) ----
void ranf_powers(unsigned long long* pw);
unsigned long long ranf_skip(unsigned long long seed, unsigned long long n);
// ran_gauss_volh on the device: out[i*m + j] for draws 2(i m + j)+1, +2 from state s0
void launch_ran_gauss(double2* out, int volh, int m, double var, unsigned long long s0, cudaStream_t s);
void launch_u_normalize(double2* u_fortran, long long nlinks, cudaStream_t s);
void launch_cold(double2* u_fortran, long long nlinks, cudaStream_t s);
void launch_conf_relax(const Geom& g, double2* gauge, cudaStream_t s);
void launch_plaquette(const Geom& g, const double2* gauge, RedScratch red, double* out, cudaStream_t s);

// ---- resident HMC pieces (hmc.cu) ----
// U <- exp(i step p) U on every link, re-unitarised (hmc_u.F90:53-67)
void launch_hmc_u(const Geom& g, double2* gauge, const double* p, double step, cudaStream_t s);
// p += s Im Tr(lambda_j U staples) (dsg.F90:28-53), s = -step beta / 3
void launch_dsg(const Geom& g, const double2* gauge, double* p, double s, cudaStream_t st);
// sum over the momentum field of (a - b)^2, or a^2 when b is null
void launch_mom_sumsq(const Geom& g, const double* a, const double* b, RedScratch red, double* out, cudaStream_t s);
// out[0] + i out[1] = <a, b> of F64 spinors
void launch_cdot(const Geom& g, const double2* a, const double2* b, RedScratch red, double* out, cudaStream_t s);
// up to kMaxDotPairs field pairs (a_j, b_j) whose <a_j, b_j> one launch computes
constexpr int kMaxDotPairs = 8;
struct FieldPairs {
  const double2* a[kMaxDotPairs];
  const double2* b[kMaxDotPairs];
};
void launch_cdot_pairs(const Geom& g, const FieldPairs& fp, int n, RedScratch red, double* out, cudaStream_t s);
// y = ay y + (are + i aim) x
void launch_caxpby(const Geom& g, double are, double aim, const double2* x, double ay, double2* y, cudaStream_t s);

}  // namespace bqcdg
