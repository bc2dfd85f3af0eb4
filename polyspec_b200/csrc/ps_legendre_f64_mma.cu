// FP64 Legendre stage for batches, contracted on the FP64 MMA (mma.sync m8n8k4).
//
// The FP64 MMA runs on the FP64 pipe at the rate of its FMAs (37 TFLOP/s measured against 33.5 for FMAs in a
// loop), but it keeps that rate: FMAs with three distinct operands reach 60-75 % of it (register reads), and the
// adjoint's sum over rings, which costs shuffles, selections and adds in ps_legendre_f64.cu, happens inside the
// MMA.  What it needs is eight columns: four maps of spin 0 (re, im) or two of spin s (four sums each).  So this
// file takes batches, and ps_legendre_f64.cu single maps and batches that do not fill the chip; the rule and both sides'
// times stand at its launchers.
//
// A warp owns 32 ring pairs.  Every lane runs the recurrence of its ring for 16 l (spin 0) or 8 l (adjoint of spin s: f
// and (-1)^l g) and drops the values into the warp's shared tile, 16 rows of 32 rings, whose columns are ordered so that
// one 16-byte read gives a lane the elements of two A operands, 8 rings x 4 l (synthesis) or 8 l x 4 rings (adjoint).
// Rows 0-7 hold the l of parity 0 (f), rows 8-15 those of parity 1 ((-1)^l g).  The spin-s synthesis owns 16 pairs, for
// 16 l, f and g in half-warps (see there).
//   synthesis spin 0: B = alm; E, O = even and odd sums, north = E + O, south = E - O.
//   synthesis spin s: B = (a+, (-1)^l a-) for f and, the same columns exchanged, for (-1)^l g; the
//                     accumulators are the north and south sums of ps_legendre_f64.cu.
//   adjoint spin 0:   B = N + S for even, N - S for odd l.
//   adjoint spin s:   B = (Z+ north, Z- south) for f, (Z+ south, Z- north) for (-1)^l g, one accumulator
//                     for both: columns T+ and (-1)^l T-.
// Synthesis: accumulators of the warp's rings stay in registers over all l; the alm of 32 l are staged for the CTA's
// four warps.  Adjoint: the B operand (phases) stays in registers over all l; per 16 l the warps' sums meet in
// shared memory and are added up in a fixed order.  What bounds it is the latency of twelve warps an SM (the B
// operand takes their registers): the MMA pipe is busy 47 % of the time (24 maps, Nside 512, lmax 1000; 48 spin-2 maps,
// Nside 128: 41 %).  Running the next tile's recurrence between one tile's MMAs (two tiles a warp) was slower, 2806 us
// for 2667: it spills, and its FMAs queue behind the MMAs.
#include <algorithm>
#include <climits>
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
template <bool SPIN>
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
            tile[j][col] = on ? f : 0.0;
            tile[8 + j][col] = on ? ((j & 1) ? -g : g) : 0.0;
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

// ------------------------------------------------------------------ synthesis, spin 0
// grid (ceil(Rh / 128), mmax+1, groups of `per` maps); per <= 4 NT
template <int NT>
__global__ void __launch_bounds__(32 * SYN_WARPS) synth0_mma_f64(
    const RingInfo* __restrict__ rings, const double* __restrict__ mnorm, const double* __restrict__ lc,
    const double* __restrict__ lg, const double2* __restrict__ alm, int64_t as, double2* __restrict__ phase, int64_t ms,
    int64_t bs, int R, int Rh, int lmax, int mmax, int B, int per) {
  next_may_start();
  constexpr int MAPS = 4 * NT, CH = 32;
  constexpr int AROW = 8 * NT + 2;  // B-operand rows l, l + 2, .. in distinct banks
  const int m = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = blockIdx.z * per, nb = min(per, B - b0);
  __shared__ __align__(16) double s_lam_[SYN_WARPS][16][SYN_ROW];
  __shared__ __align__(16) double s_cd[2][CH];
  __shared__ __align__(16) double s_a[2][CH][AROW];
  double(*s_lam)[SYN_ROW] = s_lam_[warp];
  const int wbase = (blockIdx.x * SYN_WARPS + warp) * 32;
  const int64_t base = alm_index(m, m, lmax);

  // the chunk's alm: thread -> l = l0 + lane of maps warp, warp + 4, ..
  constexpr int PER = (MAPS + SYN_WARPS - 1) / SYN_WARPS;
  double2 pa[PER];
  double pc;
  auto fetch = [&](int l0) {
    const int64_t idx = base + (l0 - m) + lane;
    const bool in = l0 + lane <= lmax;
    const double gm = in ? lg[idx] : 0.0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int b = warp + SYN_WARPS * i;
      pa[i] = in && b < nb ? cscale(alm[(b0 + b) * as + idx], gm) : make_double2(0.0, 0.0);
    }
    pc = warp == 0 && l0 + lane < lmax ? lc[idx] : 0.0;
  };
  auto stage = [&](int buf) {
    bool bad = false;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int b = warp + SYN_WARPS * i;
      if (b < MAPS) {
        *reinterpret_cast<double2*>(&s_a[buf][lane][2 * b]) = pa[i];
        bad = bad || nonfinite(pa[i]);
      }
    }
    if (warp == 0) s_cd[buf][lane] = pc;
    return bad;
  };

  fetch(m);
  Ring<false> ring;
  ring.seed(rings, wbase + lane, Rh, m, 0, mnorm, nullptr);
  double2 acc[2][4][NT];  // even, odd l
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[a][r][t] = make_double2(0.0, 0.0);
  bool force = __syncthreads_or(stage(0));
  int buf = 0;
  for (int l0 = m; l0 <= lmax; l0 += CH, buf ^= 1) {
    const bool more = l0 + CH <= lmax;
    if (more) fetch(l0 + CH);
    if (wbase < Rh) {
#pragma unroll 1
      for (int j0 = 0; j0 < CH && l0 + j0 <= lmax; j0 += 16) {
        const int mode = warp_mode(ring.k, force);
        // ring 16 h + 8 b + c in column 16 h + 2 c + b
        ring.block(&s_cd[buf][j0], s_lam, (lane & 16) + 2 * (lane & 7) + ((lane >> 3) & 1), mode);
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
            const double* brow = s_a[buf][j0 + 2 * kr + a];
#pragma unroll
            for (int t = 0; t < NT; ++t) fb[t] = brow[8 * t + (lane >> 2)];
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
              for (int r = 0; r < 4; ++r) dmma(acc[a][r][t], fa[r], fb[t]);
          }
        __syncwarp();
      }
    }
    if (more) force = __syncthreads_or(stage(buf ^ 1));
  }
  // lane: ring 8 r + lane / 4, columns 2 (lane & 3) and the next one
  const int64_t row = int64_t(mmax + 1) * B;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int rp = wbase + 8 * r + (lane >> 2), rs = R - 1 - rp;
    if (rp >= Rh) continue;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int b = 4 * t + (lane & 3);
      if (b >= nb) continue;
      const double2 e = acc[0][r][t], d = acc[1][r][t];
      const int64_t o = m * ms + (b0 + b) * bs;
      phase[rp * row + o] = cadd(e, d);
      if (rs != rp) phase[rs * row + o] = csub(e, d);
    }
  }
}

// ------------------------------------------------------------------ synthesis, spin s
// grid (ceil(Rh / 64), mmax+1, groups of `per` maps).  A warp owns 16 ring pairs: lanes 0-15 run f, lanes 16-31
// (-1)^l g, which obeys the same recurrence at -x, each with its own scale, so that all lanes do the same.
//
// Full: four columns per map, per <= 2 NT.  GRAD: alm [B][nalm], G = -alm, C = 0; then a+ = a- and the sums of both
// hemispheres follow from those over even and over odd l: two columns per map as for spin 0, per <= 4 NT, half the
// MMAs; the tile's rows are f even, f odd, g even, g odd.
//
// Sixteen rings and twelve maps fill the same accumulators as 32 rings and six maps, with half the recurrences and
// half the A operands per MMA.  24 maps, Nside 512, lmax 1000: full 7318 us before, now 6893, GRAD 5457 and 4247.
constexpr int SYNS_ROW = 20;  // row stride of the tile (doubles): as SYN_ROW
template <int NT, bool GRAD>
__global__ void __launch_bounds__(32 * SYN_WARPS) synthS_mma_f64(
    const RingInfo* __restrict__ rings, const SeedNorm* __restrict__ seednorm, const double2* __restrict__ lcd,
    const double* __restrict__ lg, const double2* __restrict__ alm, int64_t as, double2* __restrict__ phase, int64_t ms,
    int64_t bs, int R, int Rh, int lmax, int mmax, int B, int per, int64_t nalm, int spin) {
  constexpr int MAPS = GRAD ? 4 * NT : 2 * NT, CH = 32, NC = GRAD ? 1 : 2, NA = GRAD ? 4 : 2, BLK = 16;
  constexpr int AROW = 8 * NT + (GRAD ? 2 : 4);  // rows l, l + 1, .. (GRAD: l, l + 2, ..) in distinct banks
  const int m = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = blockIdx.z * per, nb = min(per, B - b0);
  __shared__ __align__(16) double s_lam_[SYN_WARPS][2 * BLK][SYNS_ROW];
  __shared__ __align__(16) double2 s_cd[2][CH];
  __shared__ __align__(16) double s_a[2][CH][AROW];
  double(*s_lam)[SYNS_ROW] = s_lam_[warp];
  const int wbase = (blockIdx.x * SYN_WARPS + warp) * 16;
  const int64_t base = alm_index(m, m, lmax);
  const int lmin = max(m, spin);

  // the chunk's alm: thread -> l = l0 + lane of maps warp, warp + 4, ..
  constexpr int PER = (MAPS + SYN_WARPS - 1) / SYN_WARPS;
  double2 pa[PER][NC], pc;
  auto fetch = [&](int l0) {
    const int64_t idx = base + (l0 - m) + lane;
    const bool in = l0 + lane <= lmax;
    const double gm = in ? lg[idx] : 0.0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int b = warp + SYN_WARPS * i;
      const bool on = in && b < nb;
      const double2 z = make_double2(0.0, 0.0), G = on ? cscale(alm[(b0 + b) * as + idx], gm) : z;
      if constexpr (GRAD) {
        pa[i][0] = G;
      } else {
        const double2 C = on ? cscale(alm[(b0 + b) * as + nalm + idx], gm) : z;
        pa[i][0] = make_double2(G.x - C.y, G.y + C.x);
        const double2 am = make_double2(G.x + C.y, G.y - C.x);
        pa[i][1] = (lane & 1) ? make_double2(-am.x, -am.y) : am;  // l - lmin has the parity of lane
      }
    }
    pc = warp == 0 && l0 + lane < lmax ? lcd[idx] : make_double2(0.0, 0.0);
  };
  auto stage = [&](int buf) {
    bool bad = false;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int b = warp + SYN_WARPS * i;
      if (b < MAPS) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          *reinterpret_cast<double2*>(&s_a[buf][lane][2 * (b * NC + c)]) = pa[i][c];
          bad = bad || nonfinite(pa[i][c]);
        }
      }
    }
    if (warp == 0) s_cd[buf][lane] = pc;
    return bad;
  };

  fetch(lmin);
  const int half = lane >> 4, rl = wbase + (lane & 15);
  const RingInfo& ri = rings[rl < Rh ? rl : 0];
  double x = ri.z, v, vp = 0.0;
  int k;
  {
    double f, g;
    seed_spin(m, spin, ri, seednorm[m], f, g, k);
    v = half ? g : f;
    if (half) x = -x;
    if (rl >= Rh) { v = 0.0; k = 0; }
  }
  double2 acc[NA][2][NT];  // GRAD: [f, g][even, odd]
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[a][r][t] = make_double2(0.0, 0.0);
  // the values of 16 l into the lane's column: ring 8 b + c in column 2 c + b
  double* col = &s_lam[BLK * half][2 * (lane & 7) + ((lane >> 3) & 1)];
  auto steps = [&](auto mode_, const double2* cd) {
    constexpr int MODE = decltype(mode_)::value;
#pragma unroll
    for (int j = 0; j < BLK; ++j) {
      const double2 c = cd[j];
      if constexpr (MODE != LEG_DEAD)
        col[(GRAD ? (j >> 1) + BLK / 2 * (j & 1) : j) * SYNS_ROW] = MODE == LEG_LIVE || k == 0 ? v : 0.0;
      const double vn = fma(fma(c.x, x, c.y), v, -vp);
      vp = v;
      v = vn;
      if constexpr (MODE != LEG_LIVE) {
        if ((j & 3) == 3) rescale(k, v, vp);
      }
    }
  };
  bool force = __syncthreads_or(stage(0));
  int buf = 0;
  for (int l0 = lmin; l0 <= lmax; l0 += CH, buf ^= 1) {
    const bool more = l0 + CH <= lmax;
    if (more) fetch(l0 + CH);
    if (wbase < Rh) {
#pragma unroll 1
      for (int j0 = 0; j0 < CH && l0 + j0 <= lmax; j0 += BLK) {
        const int mode = warp_mode(k, force);
        const double2* cd = &s_cd[buf][j0];
        if (mode == LEG_LIVE) steps(std::integral_constant<int, LEG_LIVE>{}, cd);
        else if (mode == LEG_MIXED) steps(std::integral_constant<int, LEG_MIXED>{}, cd);
        else steps(std::integral_constant<int, LEG_DEAD>{}, cd);
        if (mode == LEG_DEAD) continue;
        __syncwarp();
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int q = 0; q < BLK / 4; ++q) {
            const int kr = 4 * q + (lane & 3), odd = GRAD ? q / (BLK / 8) : 0;  // row of the tile's half a
            const double2 fa = *reinterpret_cast<const double2*>(&s_lam[a * BLK + kr][2 * (lane >> 2)]);
            const double* brow = s_a[buf][j0 + (GRAD ? 2 * (kr - odd * BLK / 2) + odd : kr)];
            double fb[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) fb[t] = brow[8 * t + (GRAD ? (lane >> 2) : ((lane >> 2) ^ (2 * a)))];
#pragma unroll
            for (int t = 0; t < NT; ++t) {
              dmma(acc[GRAD ? 2 * a + odd : a][0][t], fa.x, fb[t]);
              dmma(acc[GRAD ? 2 * a + odd : a][1][t], fa.y, fb[t]);
            }
          }
        __syncwarp();
      }
    }
    if (more) force = __syncthreads_or(stage(buf ^ 1));
  }
  // lane: ring 8 r + lane / 4, columns 2 (lane & 3) and the next one
  const int64_t row = int64_t(mmax + 1) * B * 2;
  auto put = [&](int ring, int b, double h, double2 sp, double2 sm) {  // sums S+, S- of G + iC, G - iC
    sp = cscale(sp, h);
    sm = cscale(sm, h);
    const double2 sum = cadd(sp, sm), dif = csub(sp, sm);
    const double2 q = (spin & 1) ? dif : sum, u = (spin & 1) ? sum : dif;
    const int64_t o = ring * row + m * ms + (b0 + b) * bs;
    phase[o] = GRAD ? q : make_double2(-q.x, -q.y);
    phase[o + 1] = GRAD ? make_double2(u.y, -u.x) : make_double2(-u.y, u.x);
  };
  const double hs = ((lmin + m) & 1) ? -0.5 : 0.5;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int rp = wbase + 8 * r + (lane >> 2), rs = R - 1 - rp;
    if (rp >= Rh) continue;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      // GRAD: both hemispheres in one lane; else even lanes S+ and S- of the north ring, odd lanes those of its
      // mirror (S- in the first tile)
      const int b = GRAD ? 4 * t + (lane & 3) : 2 * t + ((lane & 3) >> 1);
      const bool south = !GRAD && (lane & 1);
      if (b >= nb || (south && rs == rp)) continue;
      double2 z = make_double2(0.0, 0.0);  // alm with l < s enter only if not finite
      for (int l = m; l < min(spin, lmax + 1); ++l)
        for (int c = 0; c < NC; ++c) z = cfma(0.0, alm[(b0 + b) * as + c * nalm + base + (l - m)], z);
      if constexpr (GRAD) {
        const double2 fe = cadd(z, acc[0][r][t]), fo = acc[1][r][t], ge = cadd(z, acc[2][r][t]), go = acc[3][r][t];
        put(rp, b, 0.5, cadd(fe, fo), csub(ge, go));
        if (rs != rp) put(rs, b, hs, cadd(ge, go), csub(fe, fo));
      } else {
        const double2 s0 = cadd(z, acc[0][r][t]), s1 = cadd(z, acc[1][r][t]);
        if (south) put(rs, b, hs, s1, s0);
        else put(rp, b, 0.5, s0, s1);
      }
    }
  }
  end_after_previous();
}

// ------------------------------------------------------------------ adjoint
// grid (1, mmax+1, groups of `per` maps); per <= 4 NT (spin 0), 2 NT (spin s)
template <bool SPIN, int NT>
struct AdjShared {
  double lam[ADJ_MMA_WARPS][16][ADJ_ROW];
  // Column pairs of 16 l, as rows of l (spin s) or of the even and then the odd l (spin 0).  Rows are 16 banks apart
  // and the pairs of a row exchanged, so that neither the MMAs' layout (two rows of four pairs an access phase) nor the
  // sums' (one pair of eight rows) meets a bank twice.
  // 24 maps, Nside 512, lmax 1000, spin 0: 2950 us with plain rows (eight lanes of the sums on a bank), 2667 so.
  double2 red[2][ADJ_MMA_WARPS][16][4 * (NT | 1)];
  __device__ static int row(int l) { return SPIN ? l : 8 * (l & 1) + (l >> 1); }
  __device__ static int pair(int row, int p) { return p ^ (SPIN ? (row >> 1) & 3 : ((row >> 1) & 1) | ((row >> 2) & 2)); }
  double2 cd[2][SPIN ? 16 : 8];
  unsigned bad[ADJ_MMA_WARPS];  // maps with a phase that is not finite
  int start[ADJ_MMA_WARPS];     // first l with a value of the warp's rings above 2^-400
};
template <bool SPIN, int NT>
__global__ void __launch_bounds__(32 * ADJ_MMA_WARPS, 3) adj_mma_f64(
    const RingInfo* __restrict__ rings, const double* __restrict__ mnorm, const SeedNorm* __restrict__ seednorm,
    const double* __restrict__ lcd, const double* __restrict__ lg, const double2* __restrict__ phase, int64_t ms,
    int64_t bs, double2* __restrict__ alm, int64_t as, int R, int Rh, int lmax, int mmax, int B, int bofs, int per,
    int64_t nalm,
    int spin, double scale) {
  if constexpr (!SPIN) next_may_start();
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
    auto coef = [&](int l) {
      double2 c = make_double2(0.0, 0.0);
      if (l < lmax) {
        if constexpr (SPIN) c = reinterpret_cast<const double2*>(lcd)[base + (l - m)];
        else c.x = lcd[base + (l - m)];
      }
      return c;
    };
    auto put_coef = [&](double2* cd, double2 c) {  // of l, by thread l - l0
      if (tid < CH) {
        if constexpr (SPIN) cd[tid] = c;
        else (&cd[0].x)[tid] = c.x;
      }
    };
    // The recurrence alone, without the other warps, up to the first 16 l in which the warp has something to add: a
    // third of all (l, m, ring) lie before, and each 16 l of them took a barrier, sums of zeros and a read and write of
    // alm.  24 maps, Nside 512, lmax 1000, spin 0: 2667 us without, 2597 with it.
    int first = INT_MAX;
    if (wbase < Rh) {
      double* st = &s_lam[0][0];
      first = lmin;
      double2 c = coef(first + (lane & 15));
      while (first <= lmax && warp_mode(ring.k, force) == LEG_DEAD) {
        if (lane < CH) {
          if constexpr (SPIN) reinterpret_cast<double2*>(st)[lane] = c;
          else st[lane] = c.x;
        }
        __syncwarp();
        c = coef(first + CH + (lane & 15));
#pragma unroll
        for (int i = 0; i < (SPIN ? 2 : 1); ++i) ring.template steps<LEG_DEAD>(st + 16 * i, s_lam, 0);
        __syncwarp();
        first += CH;
      }
    }
    if (lane == 0) S.start[warp] = first;
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
    int start = lmax + 1;
#pragma unroll
    for (int w = 0; w < ADJ_MMA_WARPS; ++w) start = min(start, S.start[w]);
    if (t0 == 0) {
      for (int b = 0; b < nb; ++b)
        for (int l = lmin + tid; l < start; l += 32 * ADJ_MMA_WARPS) {
          alm[(b0 + b) * as + base + (l - m)] = make_double2(0.0, 0.0);
          if constexpr (SPIN) alm[(b0 + b) * as + nalm + base + (l - m)] = make_double2(0.0, 0.0);
        }
    }
    put_coef(S.cd[buf], coef(start + (tid & 15)));
    __syncthreads();
    for (int l0 = start; l0 <= lmax; l0 += CH, buf ^= 1) {
      const int n = min(CH, lmax - l0 + 1);
      double2 cnext = make_double2(0.0, 0.0);
      if (tid < CH) cnext = coef(l0 + CH + tid);
      // thread -> l, re / im and maps warp, warp + 4, ..; what the sums below need from memory is fetched now
      const int ls = lane >> 1, cs = lane & 1, rs = S.row(ls);
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
        if (l0 >= first) {
          // ring 8 h + 4 b + c in column 8 h + 2 c + b
          ring.block(&S.cd[buf][j0].x, s_lam, (lane & 24) + 2 * (lane & 3) + ((lane >> 2) & 1),
                     warp_mode(ring.k, force));
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
          for (int t = 0; t < NT; ++t) {
            const int r = (SPIN ? j0 : 8 * a) + (lane >> 2);
            S.red[buf][warp][r][S.pair(r, 4 * t + (lane & 3))] = d[a][t];
          }
      }
      put_coef(S.cd[buf ^ 1], cnext);
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
            tp += (&S.red[buf][w][rs][S.pair(rs, 2 * bm)].x)[cs];
            tm += (&S.red[buf][w][rs][S.pair(rs, 2 * bm + 1)].x)[cs];
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
          for (int w = 0; w < ADJ_MMA_WARPS; ++w) v += (&S.red[buf][w][rs][S.pair(rs, bm)].x)[cs];
          (&alm[(b0 + bm) * as + os].x)[cs] = old[i][0] + v * h;
        }
      }
    }
    __syncthreads();
  }
  if constexpr (SPIN) end_after_previous();
}

template <int NT>
int synth_go(const Plan& P, const double2* alm, int64_t as, double2* phase, int64_t ms, int64_t bs, int B, int per,
             cudaStream_t st) {
  const dim3 grid((P.Rh + 32 * SYN_WARPS - 1) / (32 * SYN_WARPS), P.mmax + 1, (B + per - 1) / per);
  synth0_mma_f64<NT><<<grid, 32 * SYN_WARPS, 0, st>>>(P.d_rings, P.d_mnorm0, P.d_leg_cd[0], P.d_leg_g[0], alm, as, phase,
                                                      ms, bs, P.R, P.Rh, P.lmax, P.mmax, B, per);
  PS_LAUNCH_CHECK();
  return PS_OK;
}
template <int NT, bool GRAD>
int synthS_go(const Plan& P, const double2* alm, int64_t as, double2* phase, int64_t ms, int64_t bs, int B, int per,
              int spin, bool beside, cudaStream_t st) {
  const dim3 grid((P.Rh + 16 * SYN_WARPS - 1) / (16 * SYN_WARPS), P.mmax + 1, (B + per - 1) / per);
  return launch_leg(beside, synthS_mma_f64<NT, GRAD>, grid, 32 * SYN_WARPS, 0, st, P.d_rings, P.d_seed[spin],
                    reinterpret_cast<const double2*>(P.d_leg_cd[spin]), P.d_leg_g[spin], alm, as, phase, ms, bs, P.R,
                    P.Rh, P.lmax, P.mmax, B, per, P.nalm, spin);
}
template <bool SPIN, int NT>
int adj_go(const Plan& P, const double2* phase, int64_t ms, int64_t bs, double2* alm, int64_t as, int B, int per,
           int spin, double scale, bool beside, cudaStream_t st) {
  const size_t smem = sizeof(AdjShared<SPIN, NT>);
  if (cudaFuncSetAttribute(adj_mma_f64<SPIN, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) !=
      cudaSuccess)
    return PS_ERR_CUDA;
  const int step = per * 65535;  // grid limit
  for (int bofs = 0; bofs < B; bofs += step) {
    const int z = (std::min(step, B - bofs) + per - 1) / per;
    const int rc =
        launch_leg(beside && bofs == 0, adj_mma_f64<SPIN, NT>, dim3(1, P.mmax + 1, z), 32 * ADJ_MMA_WARPS, smem, st,
                   P.d_rings, P.d_mnorm0, P.d_seed[spin], P.d_leg_cd[spin], P.d_leg_g[spin], phase, ms, bs, alm, as,
                   P.R, P.Rh, P.lmax, P.mmax, B, bofs, per, P.nalm, spin, scale);
    if (rc != PS_OK) return rc;
  }
  return PS_OK;
}

}  // namespace

// Maps per group: as few groups as possible, evenly filled; at most 12 (adjoint of spin s: 6), the most whose
// accumulators (synthesis) or B operands (adjoint) leave the registers of three CTAs an SM.  A value computed by the
// recurrence crosses shared memory twice (16 bytes) for the FMAs of all its maps, which the shared-memory path
// feeds at about half the MMA's rate for one tile of eight columns and at full rate from three on.
static int group_maps(int B, int most) {
  const int groups = (B + most - 1) / most;
  return (B + groups - 1) / groups;
}

int launch_synth_mma_f64(const Plan& P, const double2* alm, int64_t as, double2* phase, int64_t ms, int64_t bs, int B,
                         int spin, bool grad, bool beside, cudaStream_t st) {
  const int per = group_maps(B, 12);
  if (spin == 0)
    return per <= 4   ? synth_go<1>(P, alm, as, phase, ms, bs, B, per, st)
           : per <= 8 ? synth_go<2>(P, alm, as, phase, ms, bs, B, per, st)
                      : synth_go<3>(P, alm, as, phase, ms, bs, B, per, st);
  if (grad)
    return per <= 4   ? synthS_go<1, true>(P, alm, as, phase, ms, bs, B, per, spin, beside, st)
           : per <= 8 ? synthS_go<2, true>(P, alm, as, phase, ms, bs, B, per, spin, beside, st)
                      : synthS_go<3, true>(P, alm, as, phase, ms, bs, B, per, spin, beside, st);
  switch ((per + 1) / 2) {
    case 1: return synthS_go<1, false>(P, alm, as, phase, ms, bs, B, per, spin, beside, st);
    case 2: return synthS_go<2, false>(P, alm, as, phase, ms, bs, B, per, spin, beside, st);
    case 3: return synthS_go<3, false>(P, alm, as, phase, ms, bs, B, per, spin, beside, st);
    case 4: return synthS_go<4, false>(P, alm, as, phase, ms, bs, B, per, spin, beside, st);
    case 5: return synthS_go<5, false>(P, alm, as, phase, ms, bs, B, per, spin, beside, st);
    default: return synthS_go<6, false>(P, alm, as, phase, ms, bs, B, per, spin, beside, st);
  }
}

int launch_adjoint_mma_f64(const Plan& P, const double2* phase, int64_t ms, int64_t bs, double2* alm, int64_t as, int B,
                           int spin, double scale, bool beside, cudaStream_t st) {
  const int per = group_maps(B, spin == 0 ? 12 : 6), nt = (per * (spin == 0 ? 2 : 4) + 7) / 8;
  if (spin == 0)
    return nt == 1   ? adj_go<false, 1>(P, phase, ms, bs, alm, as, B, per, 0, scale, beside, st)
           : nt == 2 ? adj_go<false, 2>(P, phase, ms, bs, alm, as, B, per, 0, scale, beside, st)
                     : adj_go<false, 3>(P, phase, ms, bs, alm, as, B, per, 0, scale, beside, st);
  return nt == 1   ? adj_go<true, 1>(P, phase, ms, bs, alm, as, B, per, spin, scale, beside, st)
         : nt == 2 ? adj_go<true, 2>(P, phase, ms, bs, alm, as, B, per, spin, scale, beside, st)
                   : adj_go<true, 3>(P, phase, ms, bs, alm, as, B, per, spin, scale, beside, st);
}

}  // namespace ps
