// What the FP64 Legendre kernels share: seeds, the scaling of values too small for FP64 and how a warp treats
// them (see ps_legendre_f64.cu).
#pragma once
#include "ps_common.cuh"

namespace ps {

// ---------------------------------------------------------------- seeds
// The products of ps_common.cuh's snorm / smul / spow on positive normal values,
// with the exponent taken from the bits (frexp handles cases that do not occur here).
__device__ __forceinline__ Scaled qnorm(double x) {
  const int hi = __double2hiint(x);
  Scaled r;
  r.e = ((hi >> 20) & 0x7ff) - 1022;
  r.v = __hiloint2double((hi & 0x000fffff) | 0x3fe00000, __double2loint(x));
  return r;
}
__device__ __forceinline__ Scaled qmul(Scaled a, Scaled b) {
  Scaled r = qnorm(a.v * b.v);
  r.e += a.e + b.e;
  return r;
}
__device__ __forceinline__ Scaled qpow(double x, int n) {
  Scaled r;
  r.v = 0.5;
  r.e = 1;
  Scaled b = qnorm(x);
  while (n) {
    if (n & 1) r = qmul(r, b);
    b = qmul(b, b);
    n >>= 1;
  }
  return r;
}

__device__ __forceinline__ void seed_spin0(int m, double sth, double mnorm, double& v, int& k) {
  Scaled s = qmul(qpow(sth, m), qnorm(mnorm));
  to_kscale(s, v, k);
  if (m & 1) v = -v;
}

// Seeds of +s lam and -s lam at l = max(m, s) (Goldberg et al. 1967 with a
// single term left in the sum), with a common scale exponent k.
__device__ __forceinline__ void seed_spin(int m, int s, const RingInfo& g, SeedNorm nrm, double& f, double& gg,
                                          int& k) {
  const double sh = sqrt(0.5 * g.omz), ch = sqrt(0.5 * g.opz);
  const int lo = m < s ? m : s, hi = m < s ? s : m;
  Scaled pf = qmul(qpow(sh, hi + lo), qpow(ch, hi - lo));
  Scaled pg = qmul(qpow(sh, hi - lo), qpow(ch, hi + lo));
  const double sgn_f = (m & 1) ? -1.0 : 1.0;
  const double sgn_g = m >= s ? sgn_f : (s & 1) ? -1.0 : 1.0;
  Scaled n;
  n.v = nrm.v;
  n.e = nrm.e;
  Scaled sf = qmul(n, pf), sg = qmul(n, pg);
  Scaled big = (sf.e >= sg.e) ? sf : sg;
  double vb;
  to_kscale(big, vb, k);
  const int shift = k * SCALE_BITS;
  f = ldexp(sf.v, max(sf.e - shift, -2000)) * sgn_f;
  gg = ldexp(sg.v, max(sg.e - shift, -2000)) * sgn_g;
}

// Size tests read the exponent bits: an FP64 compare would take a slot of the FP64 pipe.
constexpr int HI_FTHRESH = (1023 + 400) << 20;
__device__ __forceinline__ bool passed(double v) { return (__double2hiint(v) & 0x7fffffff) >= HI_FTHRESH; }
__device__ __forceinline__ bool nonfinite(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }
__device__ __forceinline__ bool nonfinite(double2 v) { return nonfinite(v.x) || nonfinite(v.y); }

// Rings of a warp that is not all live are looked at every four l: c x stays below 2^8 per l, far from
// overflow.  A value with k < 0 that has grown past 2^400 moves up by one scale.
__device__ __forceinline__ void rescale(int& k, double& cur, double& prev) {
  if (k < 0 && passed(cur)) {
    cur *= PS_FSMALL;
    prev *= PS_FSMALL;
    ++k;
  }
}
__device__ __forceinline__ void rescale(int& k, double& f, double& fp, double& g, double& gp) {
  if (k < 0 && (passed(f) || passed(g))) {
    f *= PS_FSMALL;
    fp *= PS_FSMALL;
    g *= PS_FSMALL;
    gp *= PS_FSMALL;
    ++k;
  }
}

// How a warp takes the next few l: no ring of it above 2^-400 yet (recurrence only), some, or all.
enum { LEG_DEAD = 0, LEG_MIXED = 1, LEG_LIVE = 2 };
template <int RPT>
__device__ __forceinline__ int leg_mode(const int (&k)[RPT], bool force) {
  bool all = true, any = false;
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    all = all && k[i] == 0;
    any = any || k[i] == 0;
  }
  if (__all_sync(0xffffffffu, all)) return LEG_LIVE;
  return (force || __any_sync(0xffffffffu, any)) ? LEG_MIXED : LEG_DEAD;
}

// ---------------------------------------------------------------- T and (Q, U) of the same maps side by side
// The spin-0 kernels let the next launch start once all their CTAs run (programmatic dependent launch); a spin-s kernel
// launched that way (beside) fills the SMs that the last of them leave idle, and ends after they have, so that what
// follows it follows both.  It may touch nothing that the spin-0 kernel writes, and read only what was there before that
// one started.  No effect on other launches.
// T, Q, U of one map, one after the other and so: synthesis Nside 256, lmax 767 332 and 314 us, adjoint Nside 512,
// lmax 1000 1091 and 1078 us, masked CG filter at Nside 128, lmax 256 9.1 and 8.4 ms.
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void end_after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... Params, class... Args>
int launch_leg(bool beside, void (*kern)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st,
               Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = beside ? 1 : 0;
  if (cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...) == cudaSuccess) return PS_OK;
  cudaGetLastError();
  return PS_ERR_CUDA;
}

}  // namespace ps
