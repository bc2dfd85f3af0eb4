// FP64 Legendre stage for batches, contracted on the FP64 MMA (mma.sync m8n8k4).
//
// The FP64 MMA runs on the FP64 pipe at the rate of its FMAs (37 TFLOP/s measured against 33.5 for FMAs in a
// loop), but it keeps that rate: FMAs with three distinct operands reach 60-75 % of it (register reads), and the
// adjoint's sum over rings, which costs shuffles, selections and adds in ps_legendre_f64.cu, happens inside the
// MMA.  What it needs is eight columns: four maps of spin 0 (re, im) or two of spin s (four sums each).  So this
// file takes batches and ps_legendre_f64.cu single maps; the rule and both sides' times stand at its launchers.
//
// A warp owns 32 ring pairs.  Every lane runs the recurrence of its ring for 16 l (spin 0) or 8 l (spin s: f and
// (-1)^l g) and drops the values into the warp's shared tile, 16 rows of 32 rings, whose columns are ordered so that
// one 16-byte read gives a lane the elements of two A operands, 8 rings x 4 l (synthesis) or
// 8 l x 4 rings (adjoint).  Rows 0-7 hold the l of parity 0 (f), rows 8-15 those of parity 1 ((-1)^l g):
//   synthesis spin 0: B = alm; E, O = even and odd sums, north = E + O, south = E - O.
//   synthesis spin s: B = (a+, (-1)^l a-) for f and, the same columns exchanged, for (-1)^l g; the
//                     accumulators are the north and south sums of ps_legendre_f64.cu.
//   adjoint spin 0:   B = N + S for even, N - S for odd l.
//   adjoint spin s:   B = (Z+ north, Z- south) for f, (Z+ south, Z- north) for (-1)^l g, one accumulator
//                     for both: columns T+ and (-1)^l T-.
// Synthesis: accumulators of the warp's rings stay in registers over all l; the alm of 32 l are staged for the CTA's
// four warps.  Adjoint: the B operand (phases) stays in registers over all l; per 16 l the warps' sums meet in
// shared memory and are added up in a fixed order.
#include <algorithm>
#include <type_traits>

#include "ps_legendre_f64.cuh"
#include "ps_stats.cuh"

namespace ps {
namespace {

constexpr int SYN_WARPS = 4;      // 128 ring pairs per CTA
constexpr int ADJ_MMA_WARPS = 4;  // 128 ring pairs per pass of a CTA
// Row strides (doubles) of a warp's tile: the eight lanes of a 16-byte access phase read four rows of the
// synthesis' A operand, two of the adjoint's.
constexpr int SYN_ROW = 36, ADJ_ROW = 40;

__device__ __forceinline__ void dmma(double2& d, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d.x), "+d"(d.y)
               : "d"(a), "d"(b));
}
// The recurrence of one ring pair, and the next values into column `lane` of the warp's tile.
template <bool SPIN, bool GRAD = false>
struct Ring {
  double x, f, fp, g, gp;
  int k;
  __device__ __forceinline__ void seed(const RingInfo* rings, int rp, int Rh, int m, int spin, const double* mnorm,
                                       const SeedNorm* sn) {
    const RingInfo& r = rings[rp < Rh ? rp : 0];
    x = r.z;
    fp = gp = g = 0.0;
    if constexpr (SPIN) seed_spin(m, spin, r, sn[m], f, g, k);
    else seed_spin0(m, r.sth, mnorm[m], f, k);
    if (rp >= Rh) { f = g = 0.0; k = 0; }
  }
  // The values of 16 l (spin 0) or 8 l (spin s) into column `col` of the tile; cd: their coefficients.
  template <int MODE, int ROW>
  __device__ __forceinline__ void steps(const double* cd, double (*tile)[ROW], int col) {
    constexpr int N = SPIN ? 8 : 16;
#pragma unroll
    for (int j = 0; j < N; j += SPIN ? 1 : 2) {
      const double2 c = *reinterpret_cast<const double2*>(cd + (SPIN ? 2 * j : j));
#pragma unroll
      for (int h = 0; h < (SPIN ? 1 : 2); ++h) {
        if constexpr (MODE != LEG_DEAD) {
          const bool on = MODE == LEG_LIVE || k == 0;
          if constexpr (SPIN) {
            const int row = GRAD ? (j >> 1) + 4 * (j & 1) : j;
            tile[row][col] = on ? f : 0.0;
            tile[8 + row][col] = on ? ((j & 1) && !GRAD ? -g : g) : 0.0;
          } else {
            tile[8 * h + (j >> 1)][col] = on ? f : 0.0;
          }
        }
        if constexpr (SPIN) {
          const double fn = fma(fma(c.x, x, c.y), f, -fp), gn = fma(fma(c.x, x, -c.y), g, -gp);
          fp = f; f = fn;
          gp = g; g = gn;
        } else {
          const double fn = fma((h ? c.y : c.x) * x, f, -fp);
          fp = f; f = fn;
        }
      }
      if constexpr (MODE != LEG_LIVE) {
        if (SPIN ? (j & 3) == 3 : (j & 2)) {
          if constexpr (SPIN) rescale(k, f, fp, g, gp);
          else rescale(k, f, fp);
        }
      }
    }
  }
  template <int ROW>
  __device__ __forceinline__ void block(const double* cd, double (*tile)[ROW], int col, int mode) {
    if (mode == LEG_LIVE) steps<LEG_LIVE>(cd, tile, col);
    else if (mode == LEG_MIXED) steps<LEG_MIXED>(cd, tile, col);
    else steps<LEG_DEAD>(cd, tile, col);
  }
};

__device__ __forceinline__ int warp_mode(int k, bool force) {
  const int ks[1] = {k};
  return leg_mode<1>(ks, force);
}

// ------------------------------------------------------------------ synthesis
// grid (ceil(Rh / 128), mmax+1, groups of `per` maps); per <= 4 NT (spin 0 and GRAD), 2 NT (spin s)
//
// GRAD: spin s with alm [B][nalm], G = -alm, C = 0.  Then a+ = a- and the sums of both hemispheres follow from those over
// even and over odd l, a map takes two columns as for spin 0, and half the MMAs remain; the tile's rows are f even, f
// odd, g even, g odd.
template <bool SPIN, int NT, bool GRAD = false>
__global__ void __launch_bounds__(32 * SYN_WARPS) synth_mma_f64(
    const RingInfo* __restrict__ rings, const double* __restrict__ mnorm, const SeedNorm* __restrict__ seednorm,
    const double* __restrict__ lcd, const double* __restrict__ lg, const double2* __restrict__ alm, int64_t as,
    double2* __restrict__ phase, int64_t ms, int64_t bs, int R, int Rh, int lmax, int mmax, int B, int per,
    int64_t nalm,
    int spin) {
  constexpr bool FULL = SPIN && !GRAD;  // four columns per map
  constexpr int MAPS = FULL ? 2 * NT : 4 * NT, CH = 32, BLK = SPIN ? 8 : 16;
  constexpr int AROW = 8 * NT + (FULL ? 4 : 2);  // B-operand rows l, l + 1, .. (else l, l + 2, ..) in distinct banks
  const int m = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = blockIdx.z * per, nb = min(per, B - b0);
  __shared__ __align__(16) double s_lam_[SYN_WARPS][16][SYN_ROW];
  __shared__ __align__(16) double s_cd[2][CH * (SPIN ? 2 : 1)];
  __shared__ __align__(16) double s_a[2][CH][AROW];
  double(*s_lam)[SYN_ROW] = s_lam_[warp];
  const int wbase = (blockIdx.x * SYN_WARPS + warp) * 32;
  const int64_t base = alm_index(m, m, lmax);
  const int lmin = SPIN ? max(m, spin) : m;

  // the chunk's alm: thread -> l = l0 + lane of maps warp, warp + 4, ..
  constexpr int PER = (MAPS + SYN_WARPS - 1) / SYN_WARPS;
  double2 pa[PER][FULL ? 2 : 1], pc;
  auto fetch = [&](int l0) {
    const int64_t idx = base + (l0 - m) + lane;
    const bool in = l0 + lane <= lmax;
    const double gm = in ? lg[idx] : 0.0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int b = warp + SYN_WARPS * i;
      const bool on = in && b < nb;
      if constexpr (FULL) {
        const double2 z = make_double2(0.0, 0.0);
        const double2 G = on ? cscale(alm[(b0 + b) * as + idx], gm) : z;
        const double2 C = on ? cscale(alm[(b0 + b) * as + nalm + idx], gm) : z;
        pa[i][0] = make_double2(G.x - C.y, G.y + C.x);
        const double2 am = make_double2(G.x + C.y, G.y - C.x);
        pa[i][1] = (lane & 1) ? make_double2(-am.x, -am.y) : am;  // l - lmin has the parity of lane
      } else {
        pa[i][0] = on ? cscale(alm[(b0 + b) * as + idx], gm) : make_double2(0.0, 0.0);
      }
    }
    pc = make_double2(0.0, 0.0);
    if (warp == 0 && l0 + lane < lmax) {
      if constexpr (SPIN) pc = reinterpret_cast<const double2*>(lcd)[idx];
      else pc.x = lcd[idx];
    }
  };
  auto stage = [&](int buf) {
    bool bad = false;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int b = warp + SYN_WARPS * i;
      if (b < MAPS) {
#pragma unroll
        for (int c = 0; c < (FULL ? 2 : 1); ++c) {
          *reinterpret_cast<double2*>(&s_a[buf][lane][b * (FULL ? 4 : 2) + 2 * c]) = pa[i][c];
          bad = bad || nonfinite(pa[i][c]);
        }
      }
    }
    if (warp == 0) {
      if constexpr (SPIN) *reinterpret_cast<double2*>(&s_cd[buf][2 * lane]) = pc;
      else s_cd[buf][lane] = pc.x;
    }
    return bad;
  };

  fetch(lmin);
  Ring<SPIN, GRAD> ring;
  ring.seed(rings, wbase + lane, Rh, m, spin, mnorm, seednorm);
  double2 acc[GRAD ? 4 : 2][4][NT];  // GRAD: [f, g][even, odd]
#pragma unroll
  for (int a = 0; a < (GRAD ? 4 : 2); ++a)
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[a][r][t] = make_double2(0.0, 0.0);
  bool force = __syncthreads_or(stage(0));
  int buf = 0;
  for (int l0 = lmin; l0 <= lmax; l0 += CH, buf ^= 1) {
    const bool more = l0 + CH <= lmax;
    if (more) fetch(l0 + CH);
    if (wbase < Rh) {
#pragma unroll 1
      for (int j0 = 0; j0 < CH && l0 + j0 <= lmax; j0 += BLK) {
        const int mode = warp_mode(ring.k, force);
        // ring 16 h + 8 b + c in column 16 h + 2 c + b
        ring.block(&s_cd[buf][j0 * (SPIN ? 2 : 1)], s_lam, (lane & 16) + 2 * (lane & 7) + ((lane >> 3) & 1), mode);
        if (mode == LEG_DEAD) continue;
        __syncwarp();
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int kr = 4 * q + (lane & 3);  // row of the tile's half a
            double fa[4], fb[NT];
#pragma unroll
            for (int r = 0; r < 4; r += 2) {
              const double2 v = *reinterpret_cast<const double2*>(&s_lam[a * 8 + kr][8 * r + 2 * (lane >> 2)]);
              fa[r] = v.x;
              fa[r + 1] = v.y;
            }
            const double* brow = s_a[buf][j0 + (FULL ? kr : GRAD ? 2 * (lane & 3) + q : 2 * kr + a)];
#pragma unroll
            for (int t = 0; t < NT; ++t) fb[t] = brow[8 * t + (FULL ? ((lane >> 2) ^ (2 * a)) : (lane >> 2))];
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
              for (int r = 0; r < 4; ++r) dmma(acc[GRAD ? 2 * a + q : a][r][t], fa[r], fb[t]);
          }
        __syncwarp();
      }
    }
    if (more) force = __syncthreads_or(stage(buf ^ 1));
  }
  // lane: ring 8 r + lane / 4, columns 2 (lane & 3) and the next one
  const int64_t row = int64_t(mmax + 1) * B * (SPIN ? 2 : 1);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int rp = wbase + 8 * r + (lane >> 2), rs = R - 1 - rp;
    if (rp >= Rh) continue;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      if constexpr (GRAD) {
        const int b = 4 * t + (lane & 3);
        if (b >= nb) continue;
        double2 z = make_double2(0.0, 0.0);  // alm with l < s enter only if not finite
        for (int l = m; l < min(spin, lmax + 1); ++l) z = cfma(0.0, alm[(b0 + b) * as + base + (l - m)], z);
        const double2 fe = cadd(z, acc[0][r][t]), fo = acc[1][r][t], ge = cadd(z, acc[2][r][t]), go = acc[3][r][t];
        for (int south = 0; south < (rs != rp ? 2 : 1); ++south) {
          const double h = south && ((lmin + m) & 1) ? -0.5 : 0.5;
          const double2 sp = cscale(south ? csub(ge, go) : cadd(fe, fo), h);
          const double2 sm = cscale(south ? csub(fe, fo) : cadd(ge, go), h);
          const double2 sum = cadd(sp, sm), dif = csub(sp, sm);
          const double2 u = (spin & 1) ? sum : dif;
          const int64_t o = (south ? rs : rp) * row + m * ms + (b0 + b) * bs;
          phase[o] = (spin & 1) ? dif : sum;
          phase[o + 1] = make_double2(u.y, -u.x);
        }
      } else if constexpr (SPIN) {
        // even lanes: S+ and S- of the north ring, odd lanes those of its mirror (S- in the first tile)
        const int b = 2 * t + ((lane & 3) >> 1);
        const bool south = lane & 1;
        if (b >= nb || (south && rs == rp)) continue;
        double2 z = make_double2(0.0, 0.0);  // alm with l < s enter only if not finite
        for (int l = m; l < min(spin, lmax + 1); ++l)
          for (int c = 0; c < 2; ++c) z = cfma(0.0, alm[(b0 + b) * as + c * nalm + base + (l - m)], z);
        const double h = south && ((lmin + m) & 1) ? -0.5 : 0.5;
        const double2 sp = cadd(z, cscale(south ? acc[1][r][t] : acc[0][r][t], h));
        const double2 sm = cadd(z, cscale(south ? acc[0][r][t] : acc[1][r][t], h));
        const double2 sum = cadd(sp, sm), dif = csub(sp, sm);
        const double2 q = (spin & 1) ? dif : sum, u = (spin & 1) ? sum : dif;
        const int64_t o = (south ? rs : rp) * row + m * ms + (b0 + b) * bs;
        phase[o] = make_double2(-q.x, -q.y);
        phase[o + 1] = make_double2(-u.y, u.x);
      } else {
        const int b = 4 * t + (lane & 3);
        if (b >= nb) continue;
        const double2 e = acc[0][r][t], d = acc[1][r][t];
        const int64_t o = m * ms + (b0 + b) * bs;
        phase[rp * row + o] = cadd(e, d);
        if (rs != rp) phase[rs * row + o] = csub(e, d);
      }
    }
  }
}

// ------------------------------------------------------------------ adjoint
// grid (1, mmax+1, groups of `per` maps); per <= 4 NT (spin 0), 2 NT (spin s)
template <bool SPIN, int NT>
struct AdjShared {
  double lam[ADJ_MMA_WARPS][16][ADJ_ROW];
  double2 red[2][ADJ_MMA_WARPS][16][4 * NT];  // [l][column pair]
  double2 cd[2][SPIN ? 16 : 8];
  unsigned bad[ADJ_MMA_WARPS];  // maps with a phase that is not finite
};
template <bool SPIN, int NT>
__global__ void __launch_bounds__(32 * ADJ_MMA_WARPS, 3) adj_mma_f64(
    const RingInfo* __restrict__ rings, const double* __restrict__ mnorm, const SeedNorm* __restrict__ seednorm,
    const double* __restrict__ lcd, const double* __restrict__ lg, const double2* __restrict__ phase, int64_t ms,
    int64_t bs, double2* __restrict__ alm, int64_t as, int R, int Rh, int lmax, int mmax, int B, int bofs, int per,
    int64_t nalm,
    int spin, double scale) {
  constexpr int CH = 16, MAPS = SPIN ? 2 * NT : 4 * NT, ITEMS = (MAPS + ADJ_MMA_WARPS - 1) / ADJ_MMA_WARPS;
  extern __shared__ __align__(16) unsigned char adj_smem[];
  AdjShared<SPIN, NT>& S = *reinterpret_cast<AdjShared<SPIN, NT>*>(adj_smem);
  const int m = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = bofs + blockIdx.z * per, nb = min(per, B - b0);
  double(*s_lam)[ADJ_ROW] = S.lam[warp];
  const int64_t base = alm_index(m, m, lmax), row = int64_t(mmax + 1) * B * (SPIN ? 2 : 1);
  const int lmin = SPIN ? max(m, spin) : m;
  const double sgn0 = ((lmin + m) & 1) ? -1.0 : 1.0;
  int buf = 0;
  for (int t0 = 0; t0 < Rh; t0 += 32 * ADJ_MMA_WARPS) {
    const int wbase = t0 + 32 * warp;
    // B fragments: ring 4 g + (lane & 3), column lane / 4 of tile t
    double pf[2][8][NT];
    unsigned bad = 0;
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const int rp = wbase + 4 * g + (lane & 3), rs = R - 1 - rp;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int col = lane >> 2, b = SPIN ? 2 * t + (col >> 2) : 4 * t + (col >> 1);
        const bool on = rp < Rh && b < nb;
        const bool im = col & 1;
        double v0 = 0.0, v1 = 0.0;
        if (on) {
          const int64_t o = m * ms + (b0 + b) * bs;
          const double2 z = make_double2(0.0, 0.0);
          if constexpr (SPIN) {
            const double2 qn = phase[rp * row + o], un = phase[rp * row + o + 1];
            const double2 qs = rs != rp ? cscale(phase[rs * row + o], sgn0) : z;
            const double2 us = rs != rp ? cscale(phase[rs * row + o + 1], sgn0) : z;
            if (nonfinite(qn) || nonfinite(un) || nonfinite(qs) || nonfinite(us)) bad |= 1u << b;
            // columns 0, 1: Z+ = Q + i U (north for f, south for g); 2, 3: Z- = Q - i U (south for f, north for g)
            const bool minus = col & 2;
            const double2 q0 = minus ? qs : qn, u0 = minus ? us : un, q1 = minus ? qn : qs, u1 = minus ? un : us;
            const double sg = minus ? -1.0 : 1.0;
            v0 = im ? fma(sg, u0.x, q0.y) : fma(-sg, u0.y, q0.x);
            v1 = im ? fma(sg, u1.x, q1.y) : fma(-sg, u1.y, q1.x);
          } else {
            const double2 pn = phase[rp * row + o], ps = rs != rp ? phase[rs * row + o] : z;
            if (nonfinite(pn) || nonfinite(ps)) bad |= 1u << b;
            v0 = im ? pn.y + ps.y : pn.x + ps.x;
            v1 = im ? pn.y - ps.y : pn.x - ps.x;
          }
        }
        pf[0][g][t] = v0;
        pf[1][g][t] = v1;
      }
    }
    Ring<SPIN> ring;
    ring.seed(rings, wbase + lane, Rh, m, spin, mnorm, seednorm);
    bad = __reduce_or_sync(0xffffffffu, bad);
    const bool force = bad != 0;
    if (lane == 0) S.bad[warp] = bad;
    auto coef = [&](int l) {  // of l, by thread l - l0
      double2 c = make_double2(0.0, 0.0);
      if (tid < CH && l < lmax) {
        if constexpr (SPIN) c = reinterpret_cast<const double2*>(lcd)[base + (l - m)];
        else c.x = lcd[base + (l - m)];
      }
      return c;
    };
    auto put_coef = [&](int bu, double2 c) {
      if (tid < CH) {
        if constexpr (SPIN) S.cd[bu][tid] = c;
        else (&S.cd[bu][0].x)[tid] = c.x;
      }
    };
    put_coef(buf, coef(lmin + tid));
    __syncthreads();
    if (SPIN && m < spin && tid < (spin - m) * nb) {  // l < s: zero, or 0 times a phase that is not finite
      const int b = tid / (spin - m), j = tid - b * (spin - m);
      if (m + j <= lmax) {
        unsigned any = 0;
        for (int w = 0; w < ADJ_MMA_WARPS; ++w) any |= S.bad[w];
        const double z = (any >> b) & 1 ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
        for (int c = 0; c < 2; ++c) {
          double2& o = alm[(b0 + b) * as + c * nalm + base + j];
          o = t0 == 0 ? make_double2(z, z) : cadd(o, make_double2(z, z));
        }
      }
    }
    for (int l0 = lmin; l0 <= lmax; l0 += CH, buf ^= 1) {
      const int n = min(CH, lmax - l0 + 1);
      const double2 cnext = coef(l0 + CH + tid);
      // thread -> l, re / im and maps warp, warp + 4, ..; what the sums below need from memory is fetched now
      const int ls = lane >> 1, cs = lane & 1;
      const int64_t os = base + (l0 - m) + ls;
      const bool ins = ls < n;
      const double gm = ins ? lg[os] : 0.0;
      double old[ITEMS][SPIN ? 2 : 1];
      if (t0 > 0) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
          const int b = warp + ADJ_MMA_WARPS * i;
          const bool on = ins && b < nb;
          if constexpr (SPIN) {
            old[i][0] = on ? (&alm[(b0 + b) * as + os].x)[cs] : 0.0;
            old[i][1] = on ? (&alm[(b0 + b) * as + nalm + os].x)[cs ^ 1] : 0.0;
          } else {
            old[i][0] = on ? (&alm[(b0 + b) * as + os].x)[cs] : 0.0;
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
#pragma unroll
          for (int c = 0; c < (SPIN ? 2 : 1); ++c) old[i][c] = 0.0;
      }
#pragma unroll 1
      for (int j0 = 0; j0 < CH; j0 += SPIN ? 8 : 16) {
        double2 d[SPIN ? 1 : 2][NT];
#pragma unroll
        for (int a = 0; a < (SPIN ? 1 : 2); ++a)
#pragma unroll
          for (int t = 0; t < NT; ++t) d[a][t] = make_double2(0.0, 0.0);
        const int mode = wbase < Rh ? warp_mode(ring.k, force) : int(LEG_DEAD);
        // ring 8 h + 4 b + c in column 8 h + 2 c + b
        if (wbase < Rh)
          ring.block(&S.cd[buf][j0].x, s_lam, (lane & 24) + 2 * (lane & 3) + ((lane >> 2) & 1), mode);
        if (mode != LEG_DEAD) {
          __syncwarp();
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            double2 fa[4];
#pragma unroll
            for (int h = 0; h < 4; ++h)
              fa[h] = *reinterpret_cast<const double2*>(&s_lam[a * 8 + (lane >> 2)][8 * h + 2 * (lane & 3)]);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
#pragma unroll
              for (int t = 0; t < NT; ++t) dmma(d[SPIN ? 0 : a][t], fa[h].x, pf[a][2 * h][t]);
#pragma unroll
              for (int t = 0; t < NT; ++t) dmma(d[SPIN ? 0 : a][t], fa[h].y, pf[a][2 * h + 1][t]);
            }
          }
          __syncwarp();
        }
#pragma unroll
        for (int a = 0; a < (SPIN ? 1 : 2); ++a)
#pragma unroll
          for (int t = 0; t < NT; ++t)
            S.red[buf][warp][SPIN ? j0 + (lane >> 2) : 2 * (lane >> 2) + a][4 * t + (lane & 3)] = d[a][t];
      }
      put_coef(buf ^ 1, cnext);
      __syncthreads();
      const double h = gm * scale;
#pragma unroll
      for (int i = 0; i < ITEMS; ++i) {
        const int bm = warp + ADJ_MMA_WARPS * i;
        if (!ins || bm >= nb) continue;
        if constexpr (SPIN) {
          double tp = 0.0, tm = 0.0;
#pragma unroll
          for (int w = 0; w < ADJ_MMA_WARPS; ++w) {
            tp += (&S.red[buf][w][ls][2 * bm].x)[cs];
            tm += (&S.red[buf][w][ls][2 * bm + 1].x)[cs];
          }
          if (ls & 1) tm = -tm;
          const double sum = 0.5 * h * (tp + tm), dif = 0.5 * h * (tp - tm);
          // G = -(..); C = i (..): the real parts' sum is C's imaginary part, the imaginary ones', negated, its real
          const double G = (spin & 1) ? -dif : -sum, C = (spin & 1) ? sum : dif;
          (&alm[(b0 + bm) * as + os].x)[cs] = old[i][0] + G;
          (&alm[(b0 + bm) * as + nalm + os].x)[cs ^ 1] = old[i][1] + (cs ? -C : C);
        } else {
          double v = 0.0;
#pragma unroll
          for (int w = 0; w < ADJ_MMA_WARPS; ++w) v += (&S.red[buf][w][ls][bm].x)[cs];
          (&alm[(b0 + bm) * as + os].x)[cs] = old[i][0] + v * h;
        }
      }
    }
    __syncthreads();
  }
}

template <bool SPIN, int NT, bool GRAD = false>
int synth_go(const Plan& P, const double2* alm, int64_t as, double2* phase, int64_t ms, int64_t bs, int B, int per,
             int spin, cudaStream_t st) {
  const dim3 grid((P.Rh + 32 * SYN_WARPS - 1) / (32 * SYN_WARPS), P.mmax + 1, (B + per - 1) / per);
  synth_mma_f64<SPIN, NT, GRAD><<<grid, 32 * SYN_WARPS, 0, st>>>(P.d_rings, P.d_mnorm0, P.d_seed[spin], P.d_leg_cd[spin],
                                                           P.d_leg_g[spin], alm, as, phase, ms, bs, P.R, P.Rh, P.lmax,
                                                           P.mmax, B, per, P.nalm, spin);
  PS_LAUNCH_CHECK();
  return PS_OK;
}
template <bool SPIN, int NT>
int adj_go(const Plan& P, const double2* phase, int64_t ms, int64_t bs, double2* alm, int64_t as, int B, int per,
           int spin, double scale, cudaStream_t st) {
  const size_t smem = sizeof(AdjShared<SPIN, NT>);
  if (cudaFuncSetAttribute(adj_mma_f64<SPIN, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) !=
      cudaSuccess)
    return PS_ERR_CUDA;
  const int step = per * 65535;  // grid limit
  for (int bofs = 0; bofs < B; bofs += step) {
    const int z = (std::min(step, B - bofs) + per - 1) / per;
    adj_mma_f64<SPIN, NT><<<dim3(1, P.mmax + 1, z), 32 * ADJ_MMA_WARPS, smem, st>>>(
        P.d_rings, P.d_mnorm0, P.d_seed[spin], P.d_leg_cd[spin], P.d_leg_g[spin], phase, ms, bs, alm, as, P.R, P.Rh,
        P.lmax, P.mmax, B, bofs, per, P.nalm, spin, scale);
    PS_LAUNCH_CHECK();
  }
  return PS_OK;
}

}  // namespace

// Maps per group: as few groups as possible, evenly filled; at most 12 (spin 0) or 6 (spin s), the most whose
// accumulators (synthesis) or B operands (adjoint) leave the registers of three CTAs an SM.  A value computed by the
// recurrence crosses shared memory twice (16 bytes) for the FMAs of all its maps, which the shared-memory path
// feeds at about half the MMA's rate for one tile of eight columns and at full rate from three on.
static int group_maps(int B, int most) {
  const int groups = (B + most - 1) / most;
  return (B + groups - 1) / groups;
}

int launch_synth_mma_f64(const Plan& P, const double2* alm, int64_t as, double2* phase, int64_t ms, int64_t bs, int B,
                         int spin, bool grad, cudaStream_t st) {
  if (grad) {
    const int per = group_maps(B, 8);  // 24 maps, Nside 512, lmax 1000: 5457 us, with C 7318
    return per <= 4 ? synth_go<true, 1, true>(P, alm, as, phase, ms, bs, B, per, spin, st)
                    : synth_go<true, 2, true>(P, alm, as, phase, ms, bs, B, per, spin, st);
  }
  const int per = group_maps(B, spin == 0 ? 12 : 6), nt = (per * (spin == 0 ? 2 : 4) + 7) / 8;
  if (spin == 0)
    return nt == 1   ? synth_go<false, 1>(P, alm, as, phase, ms, bs, B, per, 0, st)
           : nt == 2 ? synth_go<false, 2>(P, alm, as, phase, ms, bs, B, per, 0, st)
                     : synth_go<false, 3>(P, alm, as, phase, ms, bs, B, per, 0, st);
  return nt == 1   ? synth_go<true, 1>(P, alm, as, phase, ms, bs, B, per, spin, st)
         : nt == 2 ? synth_go<true, 2>(P, alm, as, phase, ms, bs, B, per, spin, st)
                   : synth_go<true, 3>(P, alm, as, phase, ms, bs, B, per, spin, st);
}

int launch_adjoint_mma_f64(const Plan& P, const double2* phase, int64_t ms, int64_t bs, double2* alm, int64_t as, int B,
                           int spin, double scale, cudaStream_t st) {
  const int per = group_maps(B, spin == 0 ? 12 : 6), nt = (per * (spin == 0 ? 2 : 4) + 7) / 8;
  if (spin == 0)
    return nt == 1   ? adj_go<false, 1>(P, phase, ms, bs, alm, as, B, per, 0, scale, st)
           : nt == 2 ? adj_go<false, 2>(P, phase, ms, bs, alm, as, B, per, 0, scale, st)
                     : adj_go<false, 3>(P, phase, ms, bs, alm, as, B, per, 0, scale, st);
  return nt == 1   ? adj_go<true, 1>(P, phase, ms, bs, alm, as, B, per, spin, scale, st)
         : nt == 2 ? adj_go<true, 2>(P, phase, ms, bs, alm, as, B, per, spin, scale, st)
                   : adj_go<true, 3>(P, phase, ms, bs, alm, as, B, per, spin, scale, st);
}

}  // namespace ps
