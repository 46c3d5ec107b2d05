// views.cuh -- device pieces shared by the stencil kernel files: typed views
// of the type-erased field pointers (SpinorPtr, gauge void*, CloverPtr) by
// precision, and the CG scalar step that closes an iteration.
#pragma once
#include "kernels.cuh"

namespace bqcdg {

template <Prec P>
__device__ __forceinline__ SpinorView<P> sview(SpinorPtr p, int stride);
template <>
__device__ __forceinline__ SpinorView<Prec::F64> sview<Prec::F64>(SpinorPtr p, int stride) {
  return SpinorView<Prec::F64>{(double2*)p.v, stride};
}
template <>
__device__ __forceinline__ SpinorView<Prec::F32> sview<Prec::F32>(SpinorPtr p, int stride) {
  return SpinorView<Prec::F32>{(float4*)p.v, stride};
}
template <>
__device__ __forceinline__ SpinorView<Prec::F16> sview<Prec::F16>(SpinorPtr p, int stride) {
  return SpinorView<Prec::F16>{(int4*)p.v, p.norm, stride};
}

template <Prec P>
__device__ __forceinline__ GaugeView<P> gview(const void* p, const Geom& g);
template <>
__device__ __forceinline__ GaugeView<Prec::F64> gview<Prec::F64>(const void* p, const Geom& g) {
  return GaugeView<Prec::F64>{(double2*)p, g.stride, g.rec12};
}
template <>
__device__ __forceinline__ GaugeView<Prec::F32> gview<Prec::F32>(const void* p, const Geom& g) {
  return GaugeView<Prec::F32>{(float4*)p, g.stride};
}
template <>
__device__ __forceinline__ GaugeView<Prec::F16> gview<Prec::F16>(const void* p, const Geom& g) {
  return GaugeView<Prec::F16>{(short4*)p, g.stride};
}

template <Prec P>
__device__ __forceinline__ CloverView<P> cview(CloverPtr p, int stride);
template <>
__device__ __forceinline__ CloverView<Prec::F64> cview<Prec::F64>(CloverPtr p, int stride) {
  return CloverView<Prec::F64>{(double2*)p.v, stride};
}
template <>
__device__ __forceinline__ CloverView<Prec::F32> cview<Prec::F32>(CloverPtr p, int stride) {
  return CloverView<Prec::F32>{(float4*)p.v, stride};
}
template <>
__device__ __forceinline__ CloverView<Prec::F16> cview<Prec::F16>(CloverPtr p, int stride) {
  return CloverView<Prec::F16>{(int4*)p.v, p.norm, stride};
}

// Whether a right-hand side's solve has stopped, asked before chain_wait (cg
// may be null).  What is read of the flag there, while the launch that sets it
// may be in flight, is a hint and may be any value: when it is set, the kernel
// waits and asks again, and the answer is yes for certain.  When it is not, the
// solve may have stopped all the same, and the warps of a CTA may differ: a
// kernel that has a barrier or writes more than scratch reads cg->done behind
// its wait before either.  Asked only there, the flag puts a round trip to L2
// in front of a launch's gathers: int16 solves 13.5 -> 14.0 ms at 16^3x32, 242
// -> 249 ms at 32^3x64, FP64 CG at 8^4 4.35 -> 4.55 ms.
__device__ __forceinline__ bool retired(const CgScalars* cg) {
  if (!cg) return false;
  int hint;
  asm volatile("ld.global.s32 %0, [%1];" : "=r"(hint) : "l"(&cg->done) : "memory");
  if (!hint) return false;
  chain_wait();
  return cg->done != 0;
}

// |M p|^2 is known: alpha of the iteration under way
__device__ __forceinline__ void cg_set_alpha(CgScalars* cg, double paap) {
  cg->paap = paap;
  cg->alpha = cg->rtr / paap;
  cg->live = cg->iter + 1;
}

// the scalar part of one CG iteration once |r|^2 of the new residual is
// known (cg.F90:107-116), with the stop and reliable-update decisions of the
// mixed-precision solver; run by one thread of k_cg_step, or by every thread
// of k_cg_update on its own copy
__device__ __forceinline__ void cg_scalar_step(CgScalars* cg, double rtr) {
  cg->iter += 1;
  cg->rtr_old = cg->rtr;
  cg->rtr = rtr;
  cg->beta = rtr / cg->rtr_old;
  if (rtr > cg->maxr2) cg->maxr2 = rtr;
  if (!(rtr == rtr)) cg->done = 4;  // NaN: stop, reported as an error
  else if (rtr <= cg->stop_rtr) cg->done = 1;
  else if (cg->iter >= cg->maxiter) cg->done = 3;
  else if (rtr < cg->delta2 * cg->maxr2) cg->done = 2;  // reliable update (|r| < delta max|r|)
  else if (cg->ru_every > 0 && cg->iter - cg->last_ru >= cg->ru_every) cg->done = 2;  // periodic check
}

}  // namespace bqcdg
