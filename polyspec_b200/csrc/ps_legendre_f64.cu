// FP64 Legendre stage of the HEALPix SHT (the plain-precision backend).
//
// Synthesis, per order m and ring pair (theta, pi - theta):
//   spin 0:  F_m(theta) = sum_l lam_lm(theta) a_lm, split by the parity of l+m
//            so that the mirror ring is  E - O  where the north ring is E + O.
//   spin s:  with f = +s lam, g = -s lam (HEALPix conventions of
//            polyspec/base.py:247-288) and a+- = G +- i C, the sums
//            S+ = sum f a+, S- = sum g a- on the north ring and the same with
//            f and g exchanged and the sign (-1)^(l+m) on its mirror; then
//            Q = -(S+ + S-)/2, U = i (S+ - S-)/2 for even s, Q = -(S+ - S-)/2,
//            U = i (S+ + S-)/2 for odd s.
// Adjoint: the exact transpose, a_lm = sum_rings lam_lm(theta_r) P_m(r) (and the
// spin analogue), under the m-weighted alm inner product of
// polyspec/weighting.py:255, i.e. ducc0.sht.adjoint_synthesis.
//
// Recurrences: lam_l = gam_l mu_l with gam chosen so that the three-term
// recurrence keeps the unit coefficient on its second term,
//   mu_{l+1} = c_l x mu_l - mu_{l-1},   f_{l+1} = (c_l x + d_l) f_l - f_{l-1},
//   g_{l+1} = (c_l x - d_l) g_l - g_{l-1}   (f, g scaled alike)
// two FP64 instructions per l (four for f and g).  c, d and gam are tables of the
// plan (leg_tables_f64); gam multiplies the alm once, outside the ring loops.
// Seeds are scaled by 2^(800k) so that high m near the poles neither underflows
// nor loses accuracy (Reinecke & Seljebotn 2013).
//
// What bounds these kernels: the FP64 pipe (64 lanes per clock and SM; the FP64
// MMA shares it, 37 TFLOP/s either way).  Per l and ring a map needs 2 (spin 0) or
// 8 (spin s) FMAs, so for one map the recurrence is half (a third) of the work and
// everything else has to stay off that pipe: range checks compare the exponent
// bits as integers, values still below 2^-400 are not accumulated, and rings are
// kept several to a thread so that one broadcast of c and the alm from shared
// memory serves them all.
//
// Layouts: alm [ncomp][nalm] (m-major) per map, `as` elements from one map to the next; phases ring-major, the value
// of order m and map b of a ring at m ms + b bs (+ 1 for U): [R][B][mmax+1][ncomp] towards the ring transforms,
// [R][mmax+1][B][ncomp] in the calls of the Legendre stage alone.
#include <algorithm>
#include <type_traits>

#include "ps_legendre_f64.cuh"
#include "ps_legtab.h"
#include "ps_stats.cuh"

namespace ps {

constexpr int SYN_THREADS = 128;  // threads per synthesis CTA
constexpr int ADJ_LCH = 64;       // l chunk of the adjoint between two CTA barriers

// ---------------------------------------------------------------- recurrence tables
// One thread per order m, l by l (LegChain), all spins of the plan side by side, since a chain's latency is what it takes
// (four spins 43 us at lmax 47, 1.6 ms at 2048).  spin 0: cd is c [nalm]; spin s: (c, d) pairs.  Entries with l < s are
// zero.  Runs once per plan.
struct LegTables {
  double *cd[4], *gam[4];
};
__global__ void leg_tables_f64(int lmax, int mmax, LegTables t4) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x, s = blockIdx.y;
  double* cd = t4.cd[s];
  double* gam = t4.gam[s];
  if (m > mmax || !cd) return;
  const int l0 = max(m, s);
  const int64_t o = alm_index(0, m, lmax);
  for (int l = m; l < min(l0, lmax + 1); ++l) {
    cd[2 * (o + l)] = cd[2 * (o + l) + 1] = 0.0;  // l < s only for spin s
    gam[o + l] = 0.0;
  }
  LegChain t(m, s);
  for (int l = l0; l <= lmax; ++l, t.step()) {
    double c, d, g;
    t.values(c, d, g);
    if (s == 0) {
      cd[o + l] = c;
    } else {
      cd[2 * (o + l)] = c;
      cd[2 * (o + l) + 1] = d;
    }
    gam[o + l] = g;
  }
}

// =====================================================================
// synthesis, spin 0
// grid (ceil(Rh / (SYN_THREADS RPT)), mmax+1, B); a warp holds 32 RPT neighbouring ring pairs and
// stages its alm (times gam) and c itself, 32 l at a time and one chunk ahead: the warps of a CTA run at
// different speeds (fewer instructions while their rings are dead), so they share no barrier.
// A non-finite alm reaches every ring (its product with a value that counts as zero is NaN): a chunk
// that holds one takes the mixed steps on all warps.
template <int RPT>
__global__ void __launch_bounds__(SYN_THREADS) synth0_f64(const RingInfo* __restrict__ rings,
                                                           const double* __restrict__ mnorm,
                                                           const double* __restrict__ lc,
                                                           const double* __restrict__ lg,
                                                           const double2* __restrict__ alm, int64_t as,
                                                           double2* __restrict__ phase, int64_t ms, int64_t bs,
                                                           int R, int Rh, int lmax, int mmax, int B) {
  next_may_start();
  const int m = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, b = blockIdx.z;
  const int wbase = (blockIdx.x * SYN_THREADS + (tid & ~31)) * RPT, r0 = wbase + lane;
  if (wbase >= Rh) return;
  __shared__ double s_c_[SYN_THREADS / 32][2][32];
  __shared__ double2 s_alm_[SYN_THREADS / 32][2][32];
  double(*s_c)[32] = s_c_[warp];
  double2(*s_alm)[32] = s_alm_[warp];
  const int64_t base = alm_index(m, m, lmax);

  double2 pa;
  double pc;
  auto fetch = [&](int l0) {  // the chunk's alm (times gam) and c, into registers
    const int64_t idx = base + (l0 - m) + lane;
    const bool in = l0 + lane <= lmax;
    const double gm = in ? lg[idx] : 0.0;
    pc = l0 + lane < lmax ? lc[idx] : 0.0;
    pa = in ? cscale(alm[b * as + idx], gm) : make_double2(0.0, 0.0);
  };
  auto stage = [&](int buf) {  // registers -> shared memory; whether a value is not finite
    s_alm[buf][lane] = pa;
    s_c[buf][lane] = pc;
    return __any_sync(0xffffffffu, nonfinite(pa));  // also orders the stores before the warp's reads
  };

  fetch(m);
  double x[RPT], cur[RPT], prev[RPT];
  int k[RPT];
  const double mn = mnorm[m];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int rp = r0 + 32 * i;
    const RingInfo& g = rings[rp < Rh ? rp : 0];
    x[i] = g.z;
    prev[i] = 0.0;
    seed_spin0(m, g.sth, mn, cur[i], k[i]);
    if (rp >= Rh) { cur[i] = 0.0; k[i] = 0; }
  }
  double2 ae[RPT], ao[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) ae[i] = ao[i] = make_double2(0.0, 0.0);

  int buf = 0;
  for (int l0 = m; l0 <= lmax; l0 += 32, buf ^= 1) {
    const bool force = stage(buf);
    __syncwarp();
    const int n = min(32, lmax - l0 + 1);
    if (l0 + 32 <= lmax) fetch(l0 + 32);
    auto step = [&](auto mode, int j, double2 (&acc)[RPT]) {
      constexpr int MODE = decltype(mode)::value;
      const double c = s_c[buf][j];
      const double2 a = MODE != LEG_DEAD ? s_alm[buf][j] : make_double2(0.0, 0.0);
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        if (MODE != LEG_DEAD) acc[i] = cfma((MODE == LEG_LIVE || k[i] == 0) ? cur[i] : 0.0, a, acc[i]);
        const double nxt = fma(c * x[i], cur[i], -prev[i]);
        prev[i] = cur[i];
        cur[i] = nxt;
      }
    };
    auto four = [&](auto mode, int j) {  // l0 + m is even: even j have parity 0
      step(mode, j, ae);
      step(mode, j + 1, ao);
      step(mode, j + 2, ae);
      step(mode, j + 3, ao);
    };
    int j = 0;
    while (j + 4 <= n) {
      const int mode = leg_mode<RPT>(k, force);
      if (mode == LEG_LIVE) {
        for (; j + 8 <= n; j += 8) {
          four(std::integral_constant<int, LEG_LIVE>{}, j);
          four(std::integral_constant<int, LEG_LIVE>{}, j + 4);
        }
        if (j + 4 <= n) { four(std::integral_constant<int, LEG_LIVE>{}, j); j += 4; }
        break;
      }
      if (mode == LEG_DEAD) four(std::integral_constant<int, LEG_DEAD>{}, j);
      else four(std::integral_constant<int, LEG_MIXED>{}, j);
      j += 4;
#pragma unroll
      for (int i = 0; i < RPT; ++i) rescale(k[i], cur[i], prev[i]);
    }
    for (; j < n; ++j) {
      if (j & 1) step(std::integral_constant<int, LEG_MIXED>{}, j, ao);
      else step(std::integral_constant<int, LEG_MIXED>{}, j, ae);
    }
  }
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int rp = r0 + 32 * i, rs = R - 1 - rp;
    if (rp >= Rh) break;
    const int64_t o = m * ms + b * bs, ring = int64_t(mmax + 1) * B;
    phase[rp * ring + o] = cadd(ae[i], ao[i]);
    if (rs != rp) phase[rs * ring + o] = csub(ae[i], ao[i]);
  }
}

// =====================================================================
// synthesis, spin s > 0: alm [B][2][nalm] (G, C) -> phase [R][mmax+1][B][2] (Q, U)
// GRAD: alm [B][nalm], G = -alm, C = 0.  Then a+ = a- and the sums of both hemispheres follow from those over even and
// over odd l: four FMAs per l and ring instead of eight, in the same registers.
template <int RPT, bool GRAD>
__global__ void __launch_bounds__(SYN_THREADS) synthS_f64(const RingInfo* __restrict__ rings,
                                                           const SeedNorm* __restrict__ seednorm,
                                                           const double2* __restrict__ lcd,
                                                           const double* __restrict__ lg,
                                                           const double2* __restrict__ alm, int64_t as,
                                                           double2* __restrict__ phase, int64_t ms, int64_t bs,
                                                           int R, int Rh, int lmax, int mmax, int B, int64_t nalm,
                                                           int spin) {
  const int m = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, b = blockIdx.z;
  const int wbase = (blockIdx.x * SYN_THREADS + (tid & ~31)) * RPT, r0 = wbase + lane;
  if (wbase >= Rh) return;
  __shared__ double2 s_cd_[SYN_THREADS / 32][2][32];
  __shared__ double2 s_alm_[SYN_THREADS / 32][2][32][2];  // a+ = G + i C, a- = G - i C
  double2(*s_cd)[32] = s_cd_[warp];
  double2(*s_alm)[32][2] = s_alm_[warp];
  const int64_t base = alm_index(m, m, lmax);
  const int lmin = max(m, spin);

  double2 pp, pm, pc;
  auto fetch = [&](int l0) {
    const int64_t idx = base + (l0 - m) + lane;
    const bool in = l0 + lane <= lmax;
    const double gm = in ? lg[idx] : 0.0;
    pc = l0 + lane < lmax ? lcd[idx] : make_double2(0.0, 0.0);
    const double2 z = make_double2(0.0, 0.0);
    const double2 G = in ? cscale(alm[b * as + idx], gm) : z;
    if constexpr (GRAD) {
      pp = pm = G;
    } else {
      const double2 C = in ? cscale(alm[b * as + nalm + idx], gm) : z;
      pp = make_double2(G.x - C.y, G.y + C.x);
      pm = make_double2(G.x + C.y, G.y - C.x);
    }
  };
  auto stage = [&](int buf) {
    s_alm[buf][lane][0] = pp;
    if (!GRAD) s_alm[buf][lane][1] = pm;
    s_cd[buf][lane] = pc;
    return __any_sync(0xffffffffu, nonfinite(pp) || nonfinite(pm));
  };

  fetch(lmin);
  double x[RPT], f[RPT], fp[RPT], g[RPT], gp[RPT];
  int k[RPT];
  const SeedNorm sn = seednorm[m];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int rp = r0 + 32 * i;
    const RingInfo& gi = rings[rp < Rh ? rp : 0];
    x[i] = gi.z;
    fp[i] = gp[i] = 0.0;
    seed_spin(m, spin, gi, sn, f[i], g[i], k[i]);
    if (rp >= Rh) { f[i] = g[i] = 0.0; k[i] = 0; }
  }
  // sums on the north ring and, with the sign of l - lmin, on its mirror (GRAD: f and g over even, g and f over odd l)
  double2 PN[RPT], MN[RPT], PS[RPT], MS[RPT];
  {
    double2 z = make_double2(0.0, 0.0);
    // alm with l < s do not enter, unless not finite (0 times them)
    for (int l = m; l < min(spin, lmax + 1); ++l)
      for (int c = 0; c < (GRAD ? 1 : 2); ++c) z = cfma(0.0, alm[b * as + c * nalm + base + (l - m)], z);
#pragma unroll
    for (int i = 0; i < RPT; ++i) PN[i] = MN[i] = PS[i] = MS[i] = z;
  }

  int buf = 0;
  for (int l0 = lmin; l0 <= lmax; l0 += 32, buf ^= 1) {
    const bool force = stage(buf);
    __syncwarp();
    const int n = min(32, lmax - l0 + 1);
    if (l0 + 32 <= lmax) fetch(l0 + 32);
    auto step = [&](auto mode, auto odd, int j) {
      constexpr int MODE = decltype(mode)::value;
      constexpr double SG = decltype(odd)::value ? -1.0 : 1.0;
      const double2 cd = s_cd[buf][j];
      double2 ap = make_double2(0.0, 0.0), am = ap;
      if (MODE != LEG_DEAD) { ap = s_alm[buf][j][0]; am = GRAD ? ap : s_alm[buf][j][1]; }
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        if (MODE != LEG_DEAD) {
          const bool on = MODE == LEG_LIVE || k[i] == 0;
          const double vf = on ? f[i] : 0.0, vg = on ? g[i] : 0.0;
          if constexpr (!GRAD || !decltype(odd)::value) {
            PN[i] = cfma(vf, ap, PN[i]);
            MN[i] = cfma(vg, am, MN[i]);
          }
          if constexpr (!GRAD || decltype(odd)::value) {
            PS[i] = cfma(GRAD ? vg : SG * vg, ap, PS[i]);
            MS[i] = cfma(GRAD ? vf : SG * vf, am, MS[i]);
          }
        }
        const double fn = fma(fma(cd.x, x[i], cd.y), f[i], -fp[i]);
        const double gn = fma(fma(cd.x, x[i], -cd.y), g[i], -gp[i]);
        fp[i] = f[i]; f[i] = fn;
        gp[i] = g[i]; g[i] = gn;
      }
    };
    auto four = [&](auto mode, int j) {
      step(mode, std::false_type{}, j);
      step(mode, std::true_type{}, j + 1);
      step(mode, std::false_type{}, j + 2);
      step(mode, std::true_type{}, j + 3);
    };
    int j = 0;
    while (j + 4 <= n) {
      const int mode = leg_mode<RPT>(k, force);
      if (mode == LEG_LIVE) {
        for (; j + 4 <= n; j += 4) four(std::integral_constant<int, LEG_LIVE>{}, j);
        break;
      }
      if (mode == LEG_DEAD) four(std::integral_constant<int, LEG_DEAD>{}, j);
      else four(std::integral_constant<int, LEG_MIXED>{}, j);
      j += 4;
#pragma unroll
      for (int i = 0; i < RPT; ++i) rescale(k[i], f[i], fp[i], g[i], gp[i]);
    }
    for (; j < n; ++j) {
      if (j & 1) step(std::integral_constant<int, LEG_MIXED>{}, std::true_type{}, j);
      else step(std::integral_constant<int, LEG_MIXED>{}, std::false_type{}, j);
    }
  }
  const bool odd = spin & 1;
  const double ss = ((lmin + m) & 1) ? -0.5 : 0.5;
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int rp = r0 + 32 * i, rs = R - 1 - rp;
    if (rp >= Rh) break;
    if constexpr (GRAD) {
      const double2 fe = PN[i], ge = MN[i], go = PS[i], fo = MS[i];
      PN[i] = cadd(fe, fo);
      MN[i] = cadd(ge, go);
      PS[i] = csub(ge, go);
      MS[i] = csub(fe, fo);
    }
    for (int side = 0; side < (rs != rp ? 2 : 1); ++side) {
      const double h = side == 0 ? 0.5 : ss;
      const double2 sp = cscale(side == 0 ? PN[i] : PS[i], h), sm = cscale(side == 0 ? MN[i] : MS[i], h);
      const double2 sum = cadd(sp, sm), dif = csub(sp, sm);
      const double2 q = odd ? dif : sum, u = odd ? sum : dif;
      const int64_t o = (side == 0 ? rp : rs) * (int64_t(mmax + 1) * B * 2) + m * ms + b * bs;
      phase[o] = GRAD ? q : make_double2(-q.x, -q.y);
      phase[o + 1] = GRAD ? make_double2(u.y, -u.x) : make_double2(-u.y, u.x);
    }
  }
  end_after_previous();
}

// ---------------------------------------------------------------- adjoint
// One CTA per (m, map): its threads keep RPT ring pairs each, with their phases and the recurrence in
// registers, and sum over their own rings; 16 partial sums at a time (8 l of spin 0: re, im; 4 l of spin s:
// T+, T-) are then summed over the warp by halving exchanges: one FP64 add per value and thread next to the
// RPT FMAs.  In the first exchange (spin s: the first two) no selection is needed, because the lanes with bit 4
// set hold re and im (with bit 3 set: T+ and T-) exchanged from the start, so that every lane keeps its first
// half and sends its second.  The warps' sums meet in shared memory, in a fixed order, once per ADJ_LCH values
// of l, and alm are written directly: no partial sums in memory.  Rings beyond one pass of the CTA are further
// passes over l that add to the alm the CTA wrote before.
template <int H>
__device__ __forceinline__ void halve(double* v, int lane, int bit) {
  const bool up = lane & bit;
#pragma unroll
  for (int i = 0; i < H; ++i) {
    const double send = up ? v[i] : v[i + H], keep = up ? v[i + H] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
  }
}

// adjoint, spin 0: phase [R][mmax+1][B] -> alm [B][nalm].  grid (1, mmax+1, B)
template <int RPT, int NW>
__global__ void __launch_bounds__(32 * NW) adj0_f64(const RingInfo* __restrict__ rings,
                                                    const double* __restrict__ mnorm, const double* __restrict__ lc,
                                                    const double* __restrict__ lg, const double2* __restrict__ phase,
                                                    int64_t ms, int64_t bs, double2* __restrict__ alm, int64_t as,
                                                    int R, int Rh, int lmax, int mmax, int B, int bofs, double scale) {
  next_may_start();
  const int m = blockIdx.y, b = bofs + blockIdx.z, tid = threadIdx.x, nt = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
  __shared__ double2 s_red[2][NW][ADJ_LCH];
  __shared__ double s_c[2][ADJ_LCH];
  const int64_t base = alm_index(m, m, lmax);
  double2* out = alm + b * as + base;
  const double mn = mnorm[m];
  const bool up16 = lane & 16;
  int buf = 0;
  for (int t0 = 0; t0 < Rh; t0 += nt * RPT) {
    const int wbase = t0 + warp * 32 * RPT;
    double x[RPT], cur[RPT], prev[RPT];
    double2 E[RPT], O[RPT];
    int k[RPT];
    bool bad = false;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int rp = wbase + lane + 32 * i, rs = R - 1 - rp;
      const RingInfo& g = rings[rp < Rh ? rp : 0];
      double2 pn = make_double2(0.0, 0.0), ps = pn;
      if (rp < Rh) {
        const int64_t o = m * ms + b * bs, ring = int64_t(mmax + 1) * B;
        pn = phase[rp * ring + o];
        if (rs != rp) ps = phase[rs * ring + o];
      }
      E[i] = cadd(pn, ps);
      O[i] = csub(pn, ps);
      bad = bad || nonfinite(E[i]) || nonfinite(O[i]);
      if (up16) { E[i] = make_double2(E[i].y, E[i].x); O[i] = make_double2(O[i].y, O[i].x); }
      x[i] = g.z;
      prev[i] = 0.0;
      seed_spin0(m, g.sth, mn, cur[i], k[i]);
      if (rp >= Rh) { cur[i] = 0.0; k[i] = 0; }
    }
    // a phase that is not finite reaches every l (0 times it), as in the synthesis
    const bool force = __any_sync(0xffffffffu, bad);
    for (int t = tid; t < ADJ_LCH; t += nt) s_c[buf][t] = m + t < lmax ? lc[base + t] : 0.0;
    __syncthreads();
    for (int l0 = m; l0 <= lmax; l0 += ADJ_LCH, buf ^= 1) {
      const int n = min(ADJ_LCH, lmax - l0 + 1);
      for (int t = tid; t < ADJ_LCH; t += nt)
        s_c[buf ^ 1][t] = l0 + ADJ_LCH + t < lmax ? lc[base + (l0 - m) + ADJ_LCH + t] : 0.0;
#pragma unroll 1
      for (int j0 = 0; j0 < n; j0 += 8) {
        double v[16];
        auto block = [&](auto mode) {
          constexpr int MODE = decltype(mode)::value;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const double c = s_c[buf][j0 + j];
            double a0 = 0.0, a1 = 0.0;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
              if (MODE != LEG_DEAD) {
                const double w = (MODE == LEG_LIVE || k[i] == 0) ? cur[i] : 0.0;
                const double2 p = (j & 1) ? O[i] : E[i];
                a0 = fma(w, p.x, a0);
                a1 = fma(w, p.y, a1);
              }
              const double nxt = fma(c * x[i], cur[i], -prev[i]);
              prev[i] = cur[i];
              cur[i] = nxt;
            }
            if (MODE != LEG_DEAD) v[j] = a0 + __shfl_xor_sync(0xffffffffu, a1, 16);
            if (MODE != LEG_LIVE && (j & 3) == 3) {
#pragma unroll
              for (int i = 0; i < RPT; ++i) rescale(k[i], cur[i], prev[i]);
            }
          }
        };
        const int mode = wbase < Rh ? leg_mode<RPT>(k, force) : LEG_DEAD;
        double r = 0.0;
        if (mode == LEG_DEAD) {
          if (wbase < Rh) block(std::integral_constant<int, LEG_DEAD>{});
        } else {
          if (mode == LEG_LIVE) block(std::integral_constant<int, LEG_LIVE>{});
          else block(std::integral_constant<int, LEG_MIXED>{});
          halve<4>(v, lane, 8);
          halve<2>(v, lane, 4);
          halve<1>(v, lane, 2);
          r = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
        }
        if (!(lane & 1)) (&s_red[buf][warp][j0 + ((lane >> 1) & 7)].x)[lane >> 4] = r;
      }
      __syncthreads();
      for (int t = tid; t < n; t += nt) {
        double2 a = make_double2(0.0, 0.0);
        for (int w = 0; w < nw; ++w) a = cadd(a, s_red[buf][w][t]);
        const int64_t o = l0 - m + t;
        a = cscale(a, lg[base + o] * scale);
        out[o] = t0 == 0 ? a : cadd(out[o], a);
      }
    }
    __syncthreads();  // s_c of the next pass
  }
}

// adjoint, spin s: phase [R][mmax+1][B][2] (Q, U) -> alm [B][2][nalm] (G, C).  With Z+- = Q +- i U,
// T+ = sum f Z+(north) + (-1)^(l+m) g Z+(south), T- = sum g Z-(north) + (-1)^(l+m) f Z-(south):
// G = -(T+ + T-)/2, C = i (T+ - T-)/2 for even s, G = -(T+ - T-)/2, C = i (T+ + T-)/2 for odd s.
template <int RPT, int NW>
__global__ void __launch_bounds__(32 * NW) adjS_f64(const RingInfo* __restrict__ rings,
                                                    const SeedNorm* __restrict__ seednorm,
                                                    const double2* __restrict__ lcd, const double* __restrict__ lg,
                                                    const double2* __restrict__ phase, int64_t ms, int64_t bs,
                                                    double2* __restrict__ alm, int64_t as, int R, int Rh, int lmax,
                                                    int mmax,
                                                    int B, int bofs, int64_t nalm, int spin, double scale) {
  const int m = blockIdx.y, b = bofs + blockIdx.z, tid = threadIdx.x, nt = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
  __shared__ double s_red[2][NW][4 * ADJ_LCH];
  __shared__ double2 s_cd[2][ADJ_LCH];
  const int64_t base = alm_index(m, m, lmax);
  double2* outG = alm + b * as + base;
  double2* outC = outG + nalm;
  const int lmin = max(m, spin);
  const double sgn0 = ((lmin + m) & 1) ? -1.0 : 1.0;
  const SeedNorm sn = seednorm[m];
  const bool odd = spin & 1, up16 = lane & 16, up8 = lane & 8;
  const int dflip = up8 ? int(0x80000000) : 0;  // lanes with T+ and T- exchanged run g first: d changes sign
  int buf = 0;
  for (int t0 = 0; t0 < Rh; t0 += nt * RPT) {
    const int wbase = t0 + warp * 32 * RPT;
    double x[RPT], f[RPT], fp[RPT], g[RPT], gp[RPT];
    double2 ZPN[RPT], ZPS[RPT], ZMN[RPT], ZMS[RPT];
    int k[RPT];
    bool bad = false;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int rp = wbase + lane + 32 * i, rs = R - 1 - rp;
      const RingInfo& gi = rings[rp < Rh ? rp : 0];
      double2 qn = make_double2(0.0, 0.0), un = qn, qs = qn, us = qn;
      if (rp < Rh) {
        const int64_t ring = int64_t(mmax + 1) * B * 2, o = rp * ring + m * ms + b * bs;
        qn = phase[o];
        un = phase[o + 1];
        if (rs != rp) {
          const int64_t o2 = rs * ring + m * ms + b * bs;
          qs = cscale(phase[o2], sgn0);
          us = cscale(phase[o2 + 1], sgn0);
        }
      }
      bad = bad || nonfinite(qn) || nonfinite(un) || nonfinite(qs) || nonfinite(us);
      auto z = [&](double2 q, double2 u, bool plus) {  // Q + i U or Q - i U, re and im exchanged in the upper lanes
        const double2 v = plus ? make_double2(q.x - u.y, q.y + u.x) : make_double2(q.x + u.y, q.y - u.x);
        return up16 ? make_double2(v.y, v.x) : v;
      };
      ZPN[i] = z(qn, un, !up8);
      ZMN[i] = z(qn, un, up8);
      ZPS[i] = z(qs, us, !up8);
      ZMS[i] = z(qs, us, up8);
      x[i] = gi.z;
      fp[i] = gp[i] = 0.0;
      double sf, sg;
      seed_spin(m, spin, gi, sn, sf, sg, k[i]);
      f[i] = up8 ? sg : sf;
      g[i] = up8 ? sf : sg;
      if (rp >= Rh) { f[i] = g[i] = 0.0; k[i] = 0; }
    }
    const bool force = __any_sync(0xffffffffu, bad);
    for (int t = tid; t < ADJ_LCH; t += nt)
      s_cd[buf][t] = lmin + t < lmax ? lcd[base + (lmin - m) + t] : make_double2(0.0, 0.0);
    const bool anybad = __syncthreads_or(bad);
    if (m < spin && tid < spin - m && m + tid <= lmax) {  // l < s: zero, or 0 times a phase that is not finite
      const double z = anybad ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
      outG[tid] = t0 == 0 ? make_double2(z, z) : cadd(outG[tid], make_double2(z, z));
      outC[tid] = t0 == 0 ? make_double2(z, z) : cadd(outC[tid], make_double2(z, z));
    }
    for (int l0 = lmin; l0 <= lmax; l0 += ADJ_LCH, buf ^= 1) {
      const int n = min(ADJ_LCH, lmax - l0 + 1);
      for (int t = tid; t < ADJ_LCH; t += nt)
        s_cd[buf ^ 1][t] = l0 + ADJ_LCH + t < lmax ? lcd[base + (l0 - m) + ADJ_LCH + t] : make_double2(0.0, 0.0);
#pragma unroll 1
      for (int j0 = 0; j0 < n; j0 += 4) {
        double v[4];
        auto block = [&](auto mode) {
          constexpr int MODE = decltype(mode)::value;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const double2 cd = s_cd[buf][j0 + j];
            const double d = __hiloint2double(__double2hiint(cd.y) ^ dflip, __double2loint(cd.y));
            double2 tp = make_double2(0.0, 0.0), tm = tp;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
              if (MODE != LEG_DEAD) {
                const bool on = MODE == LEG_LIVE || k[i] == 0;
                const double vf = on ? f[i] : 0.0, vg = on ? g[i] : 0.0;
                tp = cfma(vf, ZPN[i], tp);
                tm = cfma(vg, ZMN[i], tm);
                tp = cfma((j & 1) ? -vg : vg, ZPS[i], tp);
                tm = cfma((j & 1) ? -vf : vf, ZMS[i], tm);
              }
              const double fn = fma(fma(cd.x, x[i], d), f[i], -fp[i]);
              const double gn = fma(fma(cd.x, x[i], -d), g[i], -gp[i]);
              fp[i] = f[i]; f[i] = fn;
              gp[i] = g[i]; g[i] = gn;
            }
            if (MODE != LEG_DEAD) {
              const double p = tp.x + __shfl_xor_sync(0xffffffffu, tp.y, 16);
              const double q = tm.x + __shfl_xor_sync(0xffffffffu, tm.y, 16);
              v[j] = p + __shfl_xor_sync(0xffffffffu, q, 8);
            }
          }
          if (MODE != LEG_LIVE) {
#pragma unroll
            for (int i = 0; i < RPT; ++i) rescale(k[i], f[i], fp[i], g[i], gp[i]);
          }
        };
        const int mode = wbase < Rh ? leg_mode<RPT>(k, force) : LEG_DEAD;
        double r = 0.0;
        if (mode == LEG_DEAD) {
          if (wbase < Rh) block(std::integral_constant<int, LEG_DEAD>{});
        } else {
          if (mode == LEG_LIVE) block(std::integral_constant<int, LEG_LIVE>{});
          else block(std::integral_constant<int, LEG_MIXED>{});
          halve<2>(v, lane, 4);
          halve<1>(v, lane, 2);
          r = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
        }
        // value: l = j0 + bits 2, 1; T- in bit 3; im in bit 4
        if (!(lane & 1)) s_red[buf][warp][4 * (j0 + ((lane >> 1) & 3)) + 2 * ((lane >> 3) & 1) + (lane >> 4)] = r;
      }
      __syncthreads();
      for (int t = tid; t < n; t += nt) {
        double2 tp = make_double2(0.0, 0.0), tm = tp;
        for (int w = 0; w < nw; ++w) {
          const double* r = &s_red[buf][w][4 * t];
          tp = cadd(tp, make_double2(r[0], r[1]));
          tm = cadd(tm, make_double2(r[2], r[3]));
        }
        const int64_t o = l0 - m + t;
        const double h = 0.5 * lg[base + o] * scale;
        const double2 sum = cscale(cadd(tp, tm), h), dif = cscale(csub(tp, tm), h);
        double2 G = odd ? dif : sum, C = odd ? sum : dif;
        G = make_double2(-G.x, -G.y);
        C = make_double2(-C.y, C.x);
        outG[o] = t0 == 0 ? G : cadd(outG[o], G);
        outC[o] = t0 == 0 ? C : cadd(outC[o], C);
      }
    }
    __syncthreads();
  }
  end_after_previous();
}

// ---------------------------------------------------------------- launchers
// algorithmic Legendre work of one transform: 4 Rh nalm flops per spin-0 map,
// 16 Rh nalm per spin-s (G, C) pair; bytes: alm in + per-ring phases out
static double leg_flops(const Plan& P, int B, int spin) {
  return double(spin == 0 ? 4 : 16) * double(P.Rh) * double(P.nalm) * B;
}
static double leg_bytes(const Plan& P, int B, int spin) {
  const double nf = double(B) * (spin == 0 ? 1 : 2);
  return nf * 16.0 * (double(P.nalm) + double(P.R) * (P.mmax + 1));
}

int launch_synth_mma_f64(const Plan& P, const double2* alm, int64_t as, double2* phase, int64_t ms, int64_t bs, int B,
                         int spin, bool grad, bool beside, cudaStream_t st);
int launch_adjoint_mma_f64(const Plan& P, const double2* phase, int64_t ms, int64_t bs, double2* alm, int64_t as, int B,
                           int spin, double scale, bool beside, cudaStream_t st);

int launch_leg_tables_f64(const Plan& P, cudaStream_t st) {
  LegTables t;
  for (int s = 0; s < 4; ++s) t.cd[s] = P.d_leg_cd[s], t.gam[s] = P.d_leg_g[s];
  leg_tables_f64<<<dim3((P.mmax + 64) / 64, 4), 64, 0, st>>>(P.lmax, P.mmax, t);
  PS_LAUNCH_CHECK();
  return PS_OK;
}

constexpr int MAX_GRID_Z = 65535;  // maps per launch

template <int RPT>
static void synth0_go(const Plan& P, const double2* alm, int64_t as, double2* phase, int64_t ms, int64_t bs, int B,
                      cudaStream_t st) {
  const dim3 grid((P.Rh + SYN_THREADS * RPT - 1) / (SYN_THREADS * RPT), P.mmax + 1, B);
  synth0_f64<RPT><<<grid, SYN_THREADS, 0, st>>>(P.d_rings, P.d_mnorm0, P.d_leg_cd[0], P.d_leg_g[0], alm, as, phase,
                                                ms, bs, P.R, P.Rh, P.lmax, P.mmax, B);
}
template <int RPT, bool GRAD>
static int synthS_go(const Plan& P, const double2* alm, int64_t as, double2* phase, int64_t ms, int64_t bs, int B,
                     int spin, bool beside, cudaStream_t st) {
  const dim3 grid((P.Rh + SYN_THREADS * RPT - 1) / (SYN_THREADS * RPT), P.mmax + 1, B);
  return launch_leg(beside, synthS_f64<RPT, GRAD>, grid, SYN_THREADS, 0, st, P.d_rings, P.d_seed[spin],
                    reinterpret_cast<const double2*>(P.d_leg_cd[spin]), P.d_leg_g[spin], alm, as, phase, ms, bs, P.R,
                    P.Rh, P.lmax, P.mmax, B, P.nalm, spin);
}

// Which kernels a batch runs on: the FP64 MMA takes maps four (spin 0) or two (spin s) at a time, and has a longer
// chain per launch; where the maps do not fill the chip the FMA kernels, a CTA for each map, are through first.  The
// line lies where the times cross: (ring pairs) (orders) (maps) of 3 2^16 and three maps for spin 0, 3 2^15 and two maps for
// spin s.  It is a rule, not a timing at run time, because the two order their sums differently (1e-15) and a call has
// to give the same bits in every process.  Measured, whole transform, FMA / MMA kernels, us:
//   spin 0: Nside 16, lmax 47: 32 maps 12.4 / 13.8; Nside 64, lmax 128: 8 maps 24.0 / 25.3, 12 27.3 / 27.4, 16 30.0 /
//     27.8; Nside 128, lmax 256: 2 maps 32.7 / 37.0, 3 36.6 / 35.8, 24 177 / 131; Nside 512, lmax 1000: 2 maps 509 / 539,
//     3 717 / 585; Nside 1024, lmax 2048: 2 maps 3042 / 3331, 3 4535 / 3528
//   spin 2: Nside 16, lmax 47: 32 maps 18.3 / 23.7; Nside 32, lmax 95: 12 maps 24.3 / 30.1, 32 43.1 / 42.2; Nside 64, lmax
//     128: 3 maps 24.1 / 25.7, 6 30.0 / 29.7, 24 78 / 63; Nside 128, lmax 256: 1 map 38.0 / 43.6, 2 52.7 / 49.0, 24 384 /
//     285; Nside 512, lmax 1000: 1 map 638 / 1007, 2 1197 / 1089
// Tile 1 forces the FMA kernels, tile 4 (spin s: 2) the MMA.  grad (C = 0), spin 2: Nside 512, lmax 1000 one map 387 us (508
// with C), 2 maps 761 / 830, 3 maps 1130 / 845; Nside 256, lmax 500 one map 64 (82), 2 maps 124 / 127, 3 maps
// 178 / 131 (Legendre stage alone): from three maps on, whatever the tile.
static bool synth_on_mma(const Plan& P, int B, int spin, bool grad) {
  if (grad) return B >= 3;
  if (P.tile[0][spin]) return P.tile[0][spin] > 1;
  const int64_t work = int64_t(P.Rh) * (P.mmax + 1) * B;
  if (B > MAX_GRID_Z) return true;  // a grid layer per map
  return spin == 0 ? B >= 3 && work >= 3 << 16 : B >= 2 && work >= 3 << 15;
}

// Rings per thread of single maps: the rings of a thread share each shared-memory broadcast, fewer keep more warps
// in flight where a plan has few rings.  Measured, one map, spin 0, one / two / four rings: Nside 1024, lmax 2048
// 1661 / 1417 / 1353 us, Nside 512, lmax 1000 212 / 187 / 184 us, Nside 256, lmax 767 70 / 71 / 81 us; spin 2 (whose
// eight sums per ring fill the registers) 4165 / 3880 / 3842 us at Nside 1024.
int launch_legendre_synth_f64(const Plan& P, const double2* alm, int64_t as, double2* phase, int64_t ms, int64_t bs,
                              int B, int spin, bool grad, bool beside, cudaStream_t st) {
  StatScope sc(PS_K_LEG_SYNTH, leg_flops(P, B, spin), leg_bytes(P, B, spin), st);
  if (spin > 0 && !P.d_seed[spin]) return PS_ERR_INVALID;
  if (synth_on_mma(P, B, spin, grad))
    return launch_synth_mma_f64(P, alm, as, phase, ms, bs, B, spin, grad, beside, st);
  if (spin == 0) {
    if (P.Rh >= 1024) synth0_go<4>(P, alm, as, phase, ms, bs, B, st);
    else if (P.Rh > 128) synth0_go<2>(P, alm, as, phase, ms, bs, B, st);
    else synth0_go<1>(P, alm, as, phase, ms, bs, B, st);
  } else if (grad) {
    return P.Rh > 128 ? synthS_go<2, true>(P, alm, as, phase, ms, bs, B, spin, beside, st)
                      : synthS_go<1, true>(P, alm, as, phase, ms, bs, B, spin, beside, st);
  } else {
    return P.Rh > 128 ? synthS_go<2, false>(P, alm, as, phase, ms, bs, B, spin, beside, st)
                      : synthS_go<1, false>(P, alm, as, phase, ms, bs, B, spin, beside, st);
  }
  PS_LAUNCH_CHECK();
  return PS_OK;
}

template <int RPT, int NW>
static void adj0_go(const Plan& P, const double2* phase, int64_t ms, int64_t bs, double2* alm, int64_t as, int B,
                    double scale, cudaStream_t st) {
  const int warps = std::min(NW, (P.Rh + 32 * RPT - 1) / (32 * RPT));
  for (int b0 = 0; b0 < B; b0 += MAX_GRID_Z)
    adj0_f64<RPT, NW><<<dim3(1, P.mmax + 1, std::min(MAX_GRID_Z, B - b0)), 32 * warps, 0, st>>>(
        P.d_rings, P.d_mnorm0, P.d_leg_cd[0], P.d_leg_g[0], phase, ms, bs, alm, as, P.R, P.Rh, P.lmax, P.mmax, B, b0,
        scale);
}
template <int RPT, int NW>
static int adjS_go(const Plan& P, const double2* phase, int64_t ms, int64_t bs, double2* alm, int64_t as, int B,
                   int spin, double scale, bool beside, cudaStream_t st) {
  const int warps = std::min(NW, (P.Rh + 32 * RPT - 1) / (32 * RPT));
  for (int b0 = 0; b0 < B; b0 += MAX_GRID_Z) {
    const int rc =
        launch_leg(beside && b0 == 0, adjS_f64<RPT, NW>, dim3(1, P.mmax + 1, std::min(MAX_GRID_Z, B - b0)), 32 * warps,
                   0, st, P.d_rings, P.d_seed[spin], reinterpret_cast<const double2*>(P.d_leg_cd[spin]),
                   P.d_leg_g[spin], phase, ms, bs, alm, as, P.R, P.Rh, P.lmax, P.mmax, B, b0, P.nalm, spin, scale);
    if (rc != PS_OK) return rc;
  }
  return PS_OK;
}

// Which kernels a batch runs on, as for the synthesis.  The MMA takes a CTA per order and twelve maps, the FMA
// kernels one per order and map: with fewer orders than SMs the MMA needs many maps to be through first.  Measured, whole
// transform, FMA / MMA kernels, us:
//   spin 0: Nside 16, lmax 47: 32 maps 12.7 / 21.9; Nside 32, lmax 95: 32 maps 26.2 / 27.6; Nside 64, lmax 128: 1 map 20.6 /
//     20.2, 4 21.5 / 20.5, 5 22.2 / 25.3, 12 29.3 / 34.2, 16 32.5 / 28.7; Nside 64, lmax 191: 3 maps 25.5 / 23.3, 4 27.1 /
//     23.3, 24 72 / 48; Nside 128, lmax 256: 3 maps 37.7 / 41.9, 4 46.1 / 43.6, 5 52.3 / 57.2, 6 61.9 / 58.5, 24 201 / 127;
//     Nside 128, lmax 383: 2 maps 48.9 / 56.3, 3 61.2 / 57.1; Nside 256, lmax 767: 2 maps 193 / 205, 3 287 / 218; Nside
//     512, lmax 1000: 2 maps 581 / 571, 3 859 / 607
//   spin 2 (the sums of two maps fill a tile), Legendre stage alone: Nside 256, lmax 767, 2 maps 430 / 326, Nside 512, 24
//     maps 16359 / 9476; one map, half a tile, 707 / 1054
// Tile 1 forces the FMA kernels of spin 0, tile 4 the MMA; spin s has no choice.
static bool adjoint_on_mma(const Plan& P, int B, int spin) {
  if (spin > 0) return B >= 2;
  if (P.tile[1][0]) return P.tile[1][0] > 1;
  const int64_t orders = P.mmax + 1, work = orders * P.Rh;
  if (orders < P.num_sms) return work * B >= 1 << 18;
  return B >= 4 || (B == 3 && work >= 90000);
}

// Rings per thread and warps per CTA.  Four rings halve the share of the warp sums and are used wherever a
// plan has enough rings for one warp of them per scheduler; a CTA of four warps passes several times over l at
// Rh > 512 but more CTAs share an SM and hide each other's barriers, eight warps keep more of the chip busy when
// there are few (m, map) pairs.  Measured, four against eight warps of four rings, one map: Nside 1024, lmax 2048
// 1898 / 1957 us (spin 0), Nside 512, lmax 1000 298 / 259 us; spin 2, <4, 4> against <2, 8>: 5280 / 5720 us,
// 706 / 759 us and, Nside 256, lmax 767, 259 / 240 us.
int launch_legendre_adjoint_f64(const Plan& P, const double2* phase, int64_t ms, int64_t bs, double2* alm, int64_t as,
                                int B, int spin, double scale, bool beside, cudaStream_t st) {
  StatScope sc(PS_K_LEG_ADJOINT, leg_flops(P, B, spin), leg_bytes(P, B, spin), st);
  if (spin > 0 && !P.d_seed[spin]) return PS_ERR_INVALID;
  if (adjoint_on_mma(P, B, spin))
    return launch_adjoint_mma_f64(P, phase, ms, bs, alm, as, B, spin, scale, beside, st);
  const int64_t ctas = int64_t(P.mmax + 1) * B;
  if (spin == 0) {
    if (P.Rh > 256 && ctas < 1500) adj0_go<4, 8>(P, phase, ms, bs, alm, as, B, scale, st);
    else if (P.Rh > 256) adj0_go<4, 4>(P, phase, ms, bs, alm, as, B, scale, st);
    else if (P.Rh > 64) adj0_go<2, 4>(P, phase, ms, bs, alm, as, B, scale, st);
    else adj0_go<1, 2>(P, phase, ms, bs, alm, as, B, scale, st);
  } else {
    if (P.Rh > 256 && ctas >= 900) return adjS_go<4, 4>(P, phase, ms, bs, alm, as, B, spin, scale, beside, st);
    if (P.Rh > 256) return adjS_go<2, 8>(P, phase, ms, bs, alm, as, B, spin, scale, beside, st);
    if (P.Rh > 64) return adjS_go<2, 4>(P, phase, ms, bs, alm, as, B, spin, scale, beside, st);
    return adjS_go<1, 2>(P, phase, ms, bs, alm, as, B, spin, scale, beside, st);
  }
  PS_LAUNCH_CHECK();
  return PS_OK;
}

}  // namespace ps
