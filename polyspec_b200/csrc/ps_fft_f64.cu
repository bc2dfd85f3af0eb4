// FP64 ring transforms of the HEALPix SHT: per ring of nphi pixels,
//   synthesis  map_j = sum_{|m| <= mmax} F_m e^{i m (phi0 + 2 pi j / nphi)}   (F_{-m} = F_m^*)
//   adjoint    P_m   = sum_j map_j e^{-i m (phi0 + 2 pi j / nphi)},  m = 0..mmax
// with the HEALPix m-aliasing (m folded modulo nphi).
//
// The two real components of a spin-s map share one complex FFT (their spectra
// are Hermitian): the synthesis transforms conj(c_a) + i conj(c_b) and reads
// map_a, map_b from the real and imaginary parts; the adjoint transforms
// x_a + i x_b and separates X_a = (Z_k + Z*_{N-k})/2, X_b = (Z_k - Z*_{N-k})/(2i).
// A spin-0 map packs a ring with its mirror ring instead (pack = 0; same length
// and phi0; the launch walks the north rings, the equator ring alone): packing two
// different maps would add the rounding of the larger to the smaller at the larger
// one's scale, which shows when batch members differ by many orders of magnitude
// (the Fisher rows of different templates do), while the two rings of one map, or
// the two components of one spin map (mixed by the Legendre stage anyway), share
// their scale.
//
// One launch takes the rings of every length up to a work length of 4096 (a second one, of
// 512-thread CTAs, the length 8192): a CTA looks up its length class and runs G = threads / T
// transforms of it, items ordered ring by ring with the fields fastest, so that the CTAs of all
// maps of a ring share in L2 the sectors of its phases (stored map-innermost).  One launch per
// class left the chip to a handful of CTAs in most of them: 10 launches of 3 to 40 us for one
// Nside 256 map.  The rings of T and of (Q, U) of the same maps share a launch too: a launch of
// one map lasts as long as its longest chain of passes, so that two of them side by side take
// little longer than one.  T, Q, U synthesis, two launches and one: Nside 16 18 and 9.5 us, 128
// 39 and 20 us, 256 94 and 78 us.
//
// The transforms are radix 8 in registers between shared-memory exchanges (one element of
// padding per eight: the stride-8 accesses are then free of bank conflicts), with a first pass of
// radix 4, 8 or 16 that makes the rest a power of 8.
//  - Power-of-two rings: Stockham (natural order in and out).  The first pass reads the folded
//    phases or pixels from global memory, the last one writes pixels.
//  - Others: Bluestein's chirp-z convolution of power-of-two length M >= 2 nphi - 1, decimation
//    in frequency, the kernel's spectrum, decimation in time; no reordering.  The upper half of
//    the input is zero and that of the output unused: the first and last pass skip them; the
//    last pass of the one, the product and the first pass of the other stay in registers.
// e^{i m phi0} = e^{i pi k / nphi} (-1)^j for m = k + j nphi (phi0 = pi / nphi or 0 on HEALPix
// rings), so the aliases of one index are summed first and rotated once; these roots and the
// chirps e^{-i pi j^2 / nphi} are tables of the plan (sincospi and 64-bit remainders per index
// took longer than the transforms).
#include <algorithm>

#include "ps_common.cuh"
#include "ps_stats.cuh"

namespace ps {

// ------------------------------------------------------------------ small DFTs in registers
constexpr double R8 = 0.70710678118654752440;   // cos(pi/4)
constexpr double C16 = 0.92387953251128675613;  // cos(pi/8)
constexpr double S16 = 0.38268343236508977173;  // sin(pi/8)

// v times -i (S < 0) or i
template <int S>
__device__ __forceinline__ double2 mul_i(double2 v) {
  return S < 0 ? make_double2(v.y, -v.x) : make_double2(-v.y, v.x);
}
// v times e^{S 2 pi i k / 16}, k a constant below 8
template <int S>
__device__ __forceinline__ double2 rot16(double2 v, int k) {
  switch (k) {
    case 0: return v;
    case 1: return make_double2(C16 * v.x - S * S16 * v.y, C16 * v.y + S * S16 * v.x);
    case 2: return make_double2(R8 * (v.x - S * v.y), R8 * (v.y + S * v.x));
    case 3: return make_double2(S16 * v.x - S * C16 * v.y, S16 * v.y + S * C16 * v.x);
    case 4: return mul_i<S>(v);
    case 5: return make_double2(-S16 * v.x - S * C16 * v.y, -S16 * v.y + S * C16 * v.x);
    case 6: return make_double2(R8 * (-v.x - S * v.y), R8 * (-v.y + S * v.x));
    default: return make_double2(-C16 * v.x - S * S16 * v.y, -C16 * v.y + S * S16 * v.x);
  }
}
__host__ __device__ constexpr int rev_bits(int k, int bits) {
  int r = 0;
  for (int b = 0; b < bits; ++b) r |= ((k >> b) & 1) << (bits - 1 - b);
  return r;
}
constexpr int log2c(int n) { return n <= 1 ? 0 : 1 + log2c(n / 2); }

// Forward DFT of R points: natural order in, position k holds frequency rev(k) out.
template <int R>
__device__ __forceinline__ void dft_dif(double2* x) {
  if constexpr (R == 2) {
    const double2 d = csub(x[0], x[1]);
    x[0] = cadd(x[0], x[1]);
    x[1] = d;
  } else {
#pragma unroll
    for (int k = 0; k < R / 2; ++k) {
      const double2 d = csub(x[k], x[k + R / 2]);
      x[k] = cadd(x[k], x[k + R / 2]);
      x[k + R / 2] = rot16<-1>(d, k * (16 / R));
    }
    dft_dif<R / 2>(x);
    dft_dif<R / 2>(x + R / 2);
  }
}
// Inverse (unscaled) DFT of R points: position k holds frequency rev(k) in, natural order out.
template <int R>
__device__ __forceinline__ void idft_dit(double2* x) {
  if constexpr (R == 2) {
    const double2 d = csub(x[0], x[1]);
    x[0] = cadd(x[0], x[1]);
    x[1] = d;
  } else {
    idft_dit<R / 2>(x);
    idft_dit<R / 2>(x + R / 2);
#pragma unroll
    for (int k = 0; k < R / 2; ++k) {
      const double2 d = rot16<1>(x[k + R / 2], k * (16 / R));
      x[k + R / 2] = csub(x[k], d);
      x[k] = cadd(x[k], d);
    }
  }
}

// Twiddles w^p_j = e^{-2 pi i p j / 2^s} of block length 2^s: the plan's table holds, level after level from
// s = 3, w^1, w^2 and w^4 for j < 2^(s-3), each contiguous in j, so that the lanes of a warp read whole lines
// (one table of the longest length, read with the stride of each level, took 32 lines per read).
__device__ __forceinline__ const double2* tw_level(const double2* __restrict__ tw, int s) {
  return tw + 3 * ((1 << (s - 3)) - 1);
}
// w[r] = w^r_j, r < 8
__device__ __forceinline__ void twiddles8(double2* w, const double2* __restrict__ tw, int s, int j) {
  const double2* L = tw_level(tw, s);
  const int q = 1 << (s - 3);
  w[1] = __ldg(&L[j]);
  w[2] = __ldg(&L[q + j]);
  w[4] = __ldg(&L[2 * q + j]);
  w[3] = cmul(w[1], w[2]);
  w[5] = cmul(w[1], w[4]);
  w[6] = cmul(w[2], w[4]);
  w[7] = cmul(w[3], w[4]);
}
// First pass of radix R = 2 H at block length 2^s, j < 2^s / R: even[r] = w^{2r}_j, r < H, and w^1_j.
template <int H>
__device__ __forceinline__ double2 twiddles_first(double2* even, const double2* __restrict__ tw, int s, int j) {
  if constexpr (H == 2) {  // j < 2^(s-2): the next level's w^2 and w^4
    const double2* L = tw_level(tw, s + 1);
    const int q = 1 << (s - 2);
    even[1] = __ldg(&L[2 * q + j]);
    return __ldg(&L[q + j]);
  } else {
    const double2* L = tw_level(tw, s);
    const int q = 1 << (s - 3);
    even[1] = __ldg(&L[q + j]);
    even[2] = __ldg(&L[2 * q + j]);
    even[3] = cmul(even[1], even[2]);
    if constexpr (H == 8) {  // w^8 is w^4 of the level below
      even[4] = __ldg(&tw_level(tw, s - 1)[q + j]);
      even[5] = cmul(even[1], even[4]);
      even[6] = cmul(even[2], even[4]);
      even[7] = cmul(even[3], even[4]);
    }
    return __ldg(&L[j]);
  }
}

__device__ __forceinline__ int pad8(int i) { return i + (i >> 3); }

// ------------------------------------------------------------------ passes over shared memory
// DIF pass of radix 8 (block length 8 q), in place.
__device__ __forceinline__ void pass_dif8(double2* a, int M, int logq, const double2* __restrict__ tw, int u,
                                          int T) {
  const int q = 1 << logq;
  for (int t = u; t < M / 8; t += T) {
    const int j = t & (q - 1), i0 = ((t >> logq) << (logq + 3)) + j;
    double2 x[8], w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = a[pad8(i0 + k * q)];
    twiddles8(w, tw, logq + 3, j);
    dft_dif<8>(x);
    a[pad8(i0)] = x[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) a[pad8(i0 + k * q)] = cmul(x[k], w[rev_bits(k, 3)]);
  }
}
// DIT pass of radix 8 (block length 8 q), in place: the inverse of pass_dif8 up to the factor 8.
__device__ __forceinline__ void pass_dit8(double2* a, int M, int logq, const double2* __restrict__ tw, int u,
                                          int T) {
  const int q = 1 << logq;
  for (int t = u; t < M / 8; t += T) {
    const int j = t & (q - 1), i0 = ((t >> logq) << (logq + 3)) + j;
    double2 x[8], w[8];
    twiddles8(w, tw, logq + 3, j);
    x[0] = a[pad8(i0)];
#pragma unroll
    for (int k = 1; k < 8; ++k) x[k] = cmul(a[pad8(i0 + k * q)], cconj(w[rev_bits(k, 3)]));
    idft_dit<8>(x);
#pragma unroll
    for (int k = 0; k < 8; ++k) a[pad8(i0 + k * q)] = x[k];
  }
}

// Bluestein convolution: in.load<H>(x, t, q) gives the inputs at t + k q, k < H, already times the chirp and zero
// from N
// on; out(j, v), j < N <= M/2, takes M times the convolution, to be multiplied by the chirp / M.  M = R1 8^n, n >= 1;
// spec is the kernel's spectrum as the middle pass reads it, [8][M/8].
template <int R1, class In, class Out>
__device__ __forceinline__ void bluestein(double2* a, int N, int M, int logM, const double2* __restrict__ spec,
                                          const double2* __restrict__ tw, int u, int T, const In& in, const Out& out) {
  constexpr int LR = log2c(R1), H = R1 / 2;
  const int q1 = M / R1;
  // first pass, the upper half of the input zero: the even frequencies are the DFT of the lower half, the odd
  // ones that of the lower half times e^{-2 pi i k / R1}
  for (int t = u; t < q1; t += T) {
    double2 x[H], y[H], we[H];
    in.template load<H>(x, t, q1);
    const double2 w1 = twiddles_first<H>(we, tw, logM, t);
#pragma unroll
    for (int k = 0; k < H; ++k) y[k] = rot16<-1>(x[k], k * (16 / R1));
    dft_dif<H>(x);
    a[pad8(t)] = x[0];
#pragma unroll
    for (int k = 1; k < H; ++k) a[pad8(t + k * q1)] = cmul(x[k], we[rev_bits(k, LR - 1)]);
    dft_dif<H>(y);
    a[pad8(t + H * q1)] = cmul(y[0], w1);
#pragma unroll
    for (int k = 1; k < H; ++k) a[pad8(t + (H + k) * q1)] = cmul(y[k], cmul(w1, we[rev_bits(k, LR - 1)]));
  }
  __syncthreads();
  int lq = logM - LR - 3;
  for (; lq > 0; lq -= 3) {
    pass_dif8(a, M, lq, tw, u, T);
    __syncthreads();
  }
  for (int t = u; t < M / 8; t += T) {
    double2 x[8], b[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) b[k] = __ldg(&spec[k * (M / 8) + t]);
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = a[9 * t + k];
    dft_dif<8>(x);
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = cmul(x[k], b[k]);
    idft_dit<8>(x);
#pragma unroll
    for (int k = 0; k < 8; ++k) a[9 * t + k] = x[k];
  }
  __syncthreads();
  for (lq = 3; lq <= logM - LR - 3; lq += 3) {
    pass_dit8(a, M, lq, tw, u, T);
    __syncthreads();
  }
  for (int t = u; t < q1; t += T) {
    double2 x[H], y[H], we[H];
    const double2 w1 = twiddles_first<H>(we, tw, logM, t);
    x[0] = a[pad8(t)];
#pragma unroll
    for (int k = 1; k < H; ++k) x[k] = cmul(a[pad8(t + k * q1)], cconj(we[rev_bits(k, LR - 1)]));
    idft_dit<H>(x);
    y[0] = cmul(a[pad8(t + H * q1)], cconj(w1));
#pragma unroll
    for (int k = 1; k < H; ++k)
      y[k] = cmul(a[pad8(t + (H + k) * q1)], cconj(cmul(w1, we[rev_bits(k, LR - 1)])));
    idft_dit<H>(y);
#pragma unroll
    for (int k = 0; k < H; ++k)
      if (t + k * q1 < N) out(t + k * q1, cadd(x[k], rot16<1>(y[k], k * (16 / R1))));
  }
}

// Stockham DFT of length M = R1 8^n; out is called by the thread that read a's elements of the same indices.
template <int R1, class In, class Out>
__device__ __forceinline__ void stockham(double2* a, int M, int logM, const double2* __restrict__ tw, int u, int T,
                                         const In& in, const Out& out) {
  constexpr int LR = log2c(R1);
  const int q1 = M / R1;
  for (int t = u; t < q1; t += T) {
    double2 x[R1];
    in.template load<R1>(x, t, q1);
    dft_dif<R1>(x);
    if (logM == LR) {
#pragma unroll
      for (int k = 0; k < R1; ++k) out(rev_bits(k, LR), x[k]);
    } else {
#pragma unroll
      for (int k = 0; k < R1; ++k) a[pad8(t * R1 + rev_bits(k, LR))] = x[k];
    }
  }
  const int q = M / 8;
  for (int ln = LR; ln < logM; ln += 3) {  // ln = log2 of the length transformed so far
    __syncthreads();
    const bool last = ln + 3 == logM;
    double2 x[2][8];  // T >= M / 16: at most two butterflies a thread
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = u + h * T;
      if (t >= q) continue;
      double2 w[8];
      twiddles8(w, tw, ln + 3, t & ((1 << ln) - 1));
      x[h][0] = a[pad8(t)];
#pragma unroll
      for (int k = 1; k < 8; ++k) x[h][k] = cmul(a[pad8(t + k * q)], w[k]);
      dft_dif<8>(x[h]);
      if (last) {
#pragma unroll
        for (int k = 0; k < 8; ++k) out(t + rev_bits(k, 3) * q, x[h][k]);
      }
    }
    if (last) break;
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = u + h * T;
      if (t >= q) continue;
      const int i0 = ((t >> ln) << (ln + 3)) + (t & ((1 << ln) - 1));
#pragma unroll
      for (int k = 0; k < 8; ++k) a[pad8(i0 + (rev_bits(k, 3) << ln))] = x[h][k];
    }
  }
}

template <class In, class Out>
__device__ __forceinline__ void ring_dft(bool blue, double2* a, int N, int M, int logM,
                                         const double2* __restrict__ spec, const double2* __restrict__ tw, int u, int T,
                                         const In& in, const Out& out) {
  const int r = logM % 3;  // the same for all transforms of a CTA
  if (blue) {
    if (r == 0) bluestein<8>(a, N, M, logM, spec, tw, u, T, in, out);
    else if (r == 1) bluestein<16>(a, N, M, logM, spec, tw, u, T, in, out);
    else bluestein<4>(a, N, M, logM, spec, tw, u, T, in, out);
  } else {
    if (r == 0) stockham<8>(a, M, logM, tw, u, T, in, out);
    else if (r == 1) stockham<16>(a, M, logM, tw, u, T, in, out);
    else stockham<4>(a, M, logM, tw, u, T, in, out);
  }
}

// ------------------------------------------------------------------ kernels
// One length class of a launch: CTAs [cta0, next class's cta0) run its `count` items, G to a CTA.
struct RingClass {
  int cta0, count, logM, logT, blue, part;
  const int* rings;
};
// The fields of one spin: nf of them, of units spin-0 maps or (packed) spin-s maps.
struct RingPart {
  int units, pack;
  int64_t nf;
  double2* phase;
  double* map;
};
constexpr int RING_CLASSES = 56;
struct RingLaunch {
  int n, mmax, R;
  int64_t npix, map_stride;  // pixels; from one map to the next
  RingPart part[2];
  const RingInfo* rings;
  const double2 *tw, *spec, *root, *chirp;
  const int64_t *spec_off, *chirp_off;
  RingClass c[RING_CLASSES];
};

// What a group of T threads works on: item -> (ring, unit) -> the two packed rows of phases and pixels.
struct RingItem {
  int N, M, logM, T, u, fa, fb, pack;
  bool blue, va, vb, turned;  // turned: phi0 = pi / N
  int64_t nf;
  double2* phase;
  double* map;
  const double2 *root, *chirp, *spec;
  int ira, irb;
  int64_t pix_a, pix_b;  // first pixels of the two rows
  double2* a;
};
__device__ __forceinline__ RingItem ring_item(const RingLaunch& L, double2* smem) {
  int ci = 0;
  while (ci + 1 < L.n && int(blockIdx.x) >= L.c[ci + 1].cta0) ++ci;
  const RingClass& c = L.c[ci];
  RingItem it;
  it.T = 1 << c.logT;
  const int G = blockDim.x >> c.logT, grp = threadIdx.x >> c.logT;
  it.u = threadIdx.x & (it.T - 1);
  const int item = (int(blockIdx.x) - c.cta0) * G + grp;
  it.logM = c.logM;
  it.M = 1 << c.logM;
  it.blue = c.blue;
  it.va = item < c.count;
  const RingPart& p = L.part[c.part];
  it.pack = p.pack;
  it.nf = p.nf;
  it.phase = p.phase;
  it.map = p.map;
  const int ring = it.va ? item / p.units : 0, unit = it.va ? item - ring * p.units : 0;
  it.ira = c.rings[ring];
  it.irb = it.pack ? it.ira : L.R - 1 - it.ira;
  const RingInfo g = L.rings[it.ira];
  it.N = g.nphi;
  it.pix_a = unit * L.map_stride + g.start;
  it.pix_b = unit * L.map_stride + (it.pack ? L.npix : 0) + L.rings[it.irb].start;
  it.turned = g.phi_num != 0;
  it.fa = it.pack ? 2 * unit : unit;
  it.fb = it.pack ? it.fa + 1 : unit;
  it.vb = it.va && (it.pack || it.irb != it.ira);
  const int i = it.N / 4;
  it.root = L.root + int64_t(2) * i * (i - 1);
  it.chirp = it.blue ? L.chirp + L.chirp_off[g.bs_slot] : nullptr;
  it.spec = it.blue ? L.spec + L.spec_off[g.bs_slot] : nullptr;
  it.a = smem + grp * (pad8(it.M) + it.T);
  return it;
}

// Phases are [R][B][mmax+1][ncomp] (ncomp 2 when packed): one transform's run contiguously in m.
__device__ __forceinline__ int64_t phase_row(const RingLaunch& L, const RingItem& it, int ring, bool second) {
  const int64_t row = int64_t(L.mmax + 1) * (it.pack ? 2 : 1);
  return (int64_t(ring) * (L.mmax + 1)) * it.nf + (it.pack ? it.fa / 2 : it.fa) * row + (it.pack && second ? 1 : 0);
}

// What a transform of the synthesis reads at index k: conj(c_a) + i conj(c_b) with
// c_k = e^{i k phi0} (sum_j step^j F_{k+jN} + step conj(sum_j step^j F_{N-k+jN})), times the chirp.
struct SynthIn {
  const double2 *pa, *pb, *root, *chirp;
  int N, mmax, ms;
  double step;  // e^{i N phi0} = +-1
  bool va, vb, blue;

  // sums over the aliases m0, m0 + dm, ... of ds^j F_m, times sg
  __device__ __forceinline__ void sum(int m0, int dm, double sg, double ds, double2& sa, double2& sb) const {
    for (int m = m0; m <= mmax; m += dm, sg *= ds) {
      sa = cfma(sg, __ldg(&pa[int64_t(m) * ms]), sa);
      if (vb) sb = cfma(sg, __ldg(&pb[int64_t(m) * ms]), sb);
    }
  }
  __device__ __forceinline__ double2 combine(int k, double2 ca, double2 cb) const {
    // (also where the rotation is 1: a part that is not finite makes its complex product so)
    const double2 e = step < 0.0 ? __ldg(&root[k]) : make_double2(1.0, 0.0);
    ca = cmul(ca, e);
    cb = cmul(cb, e);
    // a real field keeps only Re(c_0); it must not leak into the partner field of the pair
    if (k == 0) ca.y = cb.y = 0.0;
    const double2 v = make_double2(ca.x + cb.y, cb.x - ca.y);
    return blue ? cmul(v, __ldg(&chirp[k])) : v;
  }
  // x[i] = input at t + i q (zero from N on).  The first aliases of a few indices are loaded together, further
  // ones (rings with N <= mmax) in loops.
  template <int K>
  __device__ __forceinline__ void load(double2* x, int t, int q) const {
    constexpr int C = K < 2 ? K : 2;
    const double2 z = make_double2(0.0, 0.0);
#pragma unroll
    for (int c = 0; c < K; c += C) {
      double2 a1[C], a2[C], b1[C], b2[C];
#pragma unroll
      for (int i = 0; i < C; ++i) {
        const int k = t + (c + i) * q, k2 = k == 0 ? N : N - k;
        const bool on = va && k < N, h1 = on && k <= mmax, h2 = on && k2 <= mmax;
        a1[i] = h1 ? __ldg(&pa[int64_t(k) * ms]) : z;
        b1[i] = h1 && vb ? __ldg(&pb[int64_t(k) * ms]) : z;
        a2[i] = h2 ? __ldg(&pa[int64_t(k2) * ms]) : z;
        b2[i] = h2 && vb ? __ldg(&pb[int64_t(k2) * ms]) : z;
      }
      if (mmax >= N) {
#pragma unroll
        for (int i = 0; i < C; ++i) {
          const int k = t + (c + i) * q, k2 = k == 0 ? N : N - k;
          if (!va || k >= N) continue;
          sum(k + N, N, step, step, a1[i], b1[i]);
          sum(k2 + N, N, step, step, a2[i], b2[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < C; ++i) {
        const int k = t + (c + i) * q;
        x[c + i] = k < N ? combine(k, cfma(step, cconj(a2[i]), a1[i]), cfma(step, cconj(b2[i]), b1[i])) : z;
      }
    }
  }
};

// inputs already folded, in shared memory
struct PartIn {
  const double2* part;
  int N;
  template <int K>
  __device__ __forceinline__ void load(double2* x, int t, int q) const {
#pragma unroll
    for (int i = 0; i < K; ++i) x[i] = t + i * q < N ? part[t + i * q] : make_double2(0.0, 0.0);
  }
};

// synthesis: phase -> maps, or (PAIR, packed) complex maps Q + iU at map and Q - iU at minus
template <int NT, bool PAIR>
__global__ void __launch_bounds__(NT, 512 / NT) ring_synth_f64(const __grid_constant__ RingLaunch L,
                                                               double2* __restrict__ minus) {
  extern __shared__ double2 smem[];
  const RingItem it = ring_item(L, smem);
  const int N = it.N, T = it.T, u = it.u;
  SynthIn in;
  in.pa = it.phase + phase_row(L, it, it.ira, false);
  in.pb = it.phase + phase_row(L, it, it.irb, true);
  in.ms = it.pack ? 2 : 1;
  in.root = it.root;
  in.chirp = it.chirp;
  in.N = N;
  in.mmax = L.mmax;
  in.step = it.turned ? -1.0 : 1.0;
  in.va = it.va;
  in.vb = it.vb;
  in.blue = it.blue;
  double* oa = it.map + it.pix_a;
  double* ob = it.map + it.pix_b;
  double2* op = reinterpret_cast<double2*>(it.map) + it.pix_a;
  double2* om = minus + it.pix_a;
  const double inv = 1.0 / double(it.M);
  auto out = [&](int j, double2 y) {
    if (it.blue) y = cscale(cmul(y, __ldg(&it.chirp[j])), inv);
    if constexpr (PAIR) {
      if (it.va) {
        op[j] = y;
        om[j] = cconj(y);
      }
    } else {
      if (it.va) oa[j] = y.x;
      if (it.vb) ob[j] = y.y;
    }
  };
  if (T >= (it.blue ? it.M / 2 : it.M)) {
    // short rings (every ring of the class has at most T pixels): the aliases of each index are shared by
    // T / N threads and added up in order
    double2* part = it.a + pad8(it.M);
    const double2 z = make_double2(0.0, 0.0);
    const int rep = T / N, k = u % N, p = u / N;
    double2 a1 = z, a2 = z, b1 = z, b2 = z;
    if (it.va && p < rep) {
      const double sg = (p & 1) ? in.step : 1.0, ds = (rep & 1) ? in.step : 1.0;
      in.sum(k + p * N, rep * N, sg, ds, a1, b1);
      in.sum((k == 0 ? N : N - k) + p * N, rep * N, sg, ds, a2, b2);
    }
    const double2 ca = cfma(in.step, cconj(a2), a1), cb = cfma(in.step, cconj(b2), b1);
    double2 ta = z, tb = z;
    part[u] = ca;
    __syncthreads();
    if (u < N)
      for (int r = 0; r < rep; ++r) ta = cadd(ta, part[u + r * N]);
    __syncthreads();
    part[u] = cb;
    __syncthreads();
    if (u < N)
      for (int r = 0; r < rep; ++r) tb = cadd(tb, part[u + r * N]);
    __syncthreads();
    if (u < N) part[u] = in.combine(u, ta, tb);
    __syncthreads();
    ring_dft(it.blue, it.a, N, it.M, it.logM, it.spec, L.tw, u, T, PartIn{part, N}, out);
  } else {
    ring_dft(it.blue, it.a, N, it.M, it.logM, it.spec, L.tw, u, T, in, out);
  }
}

template <bool PAIR>
struct AdjointIn {
  const double *ia, *ib;
  const double2 *ip, *im;
  const double2* chirp;
  int N;
  bool va, vb, blue;
  template <int K>
  __device__ __forceinline__ void load(double2* x, int t, int q) const {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int j = t + i * q;
      if constexpr (PAIR) {
        const double2 z = make_double2(0.0, 0.0), p = va && j < N ? __ldg(&ip[j]) : z, n = va && j < N ? __ldg(&im[j]) : z;
        x[i] = make_double2(0.5 * (p.x + n.x), 0.5 * (p.y - n.y));
      } else {
        x[i] = make_double2(va && j < N ? __ldg(&ia[j]) : 0.0, vb && j < N ? __ldg(&ib[j]) : 0.0);
      }
    }
    if (blue) {
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (t + i * q < N) x[i] = cmul(x[i], __ldg(&chirp[t + i * q]));
    }
  }
};

// adjoint: maps, or (PAIR, packed) Q = Re (p + n) / 2, U = Im (p - n) / 2 of the complex maps p and n = minus -> phase
template <int NT, bool PAIR>
__global__ void __launch_bounds__(NT, 512 / NT) ring_adjoint_f64(const __grid_constant__ RingLaunch L,
                                                                 const double2* __restrict__ minus) {
  extern __shared__ double2 smem[];
  const RingItem it = ring_item(L, smem);
  const int N = it.N, mmax = L.mmax, T = it.T, u = it.u;
  const AdjointIn<PAIR> in{it.map + it.pix_a, it.map + it.pix_b, reinterpret_cast<const double2*>(it.map) + it.pix_a,
                           minus + it.pix_a, it.chirp, N, it.va, it.vb, it.blue};
  const double inv = 1.0 / double(it.M);
  auto out = [&](int k, double2 y) {
    if (it.blue) y = cscale(cmul(y, __ldg(&it.chirp[k])), inv);
    it.a[pad8(k)] = y;
  };
  ring_dft(it.blue, it.a, N, it.M, it.logM, it.spec, L.tw, u, T, in, out);
  __syncthreads();
  if (!it.va) return;
  const int ms = it.pack ? 2 : 1;
  double2* pa = it.phase + phase_row(L, it, it.ira, false);
  double2* pb = it.phase + phase_row(L, it, it.irb, true);
  for (int m = u; m <= mmax; m += T) {
    const int j = m < N ? 0 : m / N, k = m - j * N;
    const double2 z = it.a[pad8(k)], z2 = cconj(it.a[pad8(k == 0 ? 0 : N - k)]);
    double2 xa = make_double2(0.5 * (z.x + z2.x), 0.5 * (z.y + z2.y));
    double2 xb = make_double2(0.5 * (z.y - z2.y), -0.5 * (z.x - z2.x));  // (z - z2) / (2i)
    double2 e = make_double2(1.0, 0.0);
    if (it.turned) {
      e = cconj(__ldg(&it.root[k]));
      if (j & 1) e = make_double2(-e.x, -e.y);
    }
    xa = cmul(xa, e);
    xb = cmul(xb, e);
    pa[int64_t(m) * ms] = xa;
    if (it.vb) pb[int64_t(m) * ms] = xb;
  }
}

// ------------------------------------------------------------------ launch
// Threads per transform: 16 points each, and no fewer than 1/16 of the orders (short rings fold many
// aliases).  Every class then takes about the shared memory of one 4096-point transform per 256 threads.
static int ring_logT(int logM, int mmax, int nt) {
  int t = 5;
  while ((1 << t) < nt && ((1 << t) * 16 < (1 << logM) || (1 << t) * 16 < mmax + 1)) ++t;
  return t;
}

template <class Launch>
static int ring_launches(const Plan& P, const RingClassList* cls, int ncls, int64_t map_stride, const RingPart* part,
                         int nparts, Launch go) {
  RingLaunch L;
  L.mmax = P.mmax; L.R = P.R; L.npix = P.npix; L.map_stride = map_stride; L.rings = P.d_rings;
  L.tw = P.d_twiddle; L.spec = P.d_bs_spec; L.spec_off = P.d_bs_off;
  L.root = P.d_root; L.chirp = P.d_chirp; L.chirp_off = P.d_chirp_off;
  for (int p = 0; p < nparts; ++p) L.part[p] = part[p];
  for (int big = 1; big >= 0; --big) {  // work length 8192 first, then all others, longest first
    const int nt = big ? 512 : 256;
    size_t smem = 0;
    int64_t ctas = 0;
    L.n = 0;
    for (int i = 0; i < ncls; ++i) {
      const RingClassList& c = cls[i];
      if ((c.logM > 12) != (big == 1)) continue;
      for (int p = nparts - 1; p >= 0; --p) {
        const int count = part[p].pack ? c.count : c.count_n;
        if (count == 0) continue;
        if (L.n == RING_CLASSES) return PS_ERR_UNSUPPORTED;
        RingClass& r = L.c[L.n++];
        r.cta0 = int(ctas);
        r.logM = c.logM;
        r.logT = ring_logT(c.logM, P.mmax, nt);
        r.blue = c.blue;
        r.part = p;
        r.rings = part[p].pack ? c.rings : c.rings_n;
        const int64_t items = int64_t(count) * part[p].units, G = nt >> r.logT;
        if (items > 0x7fffffff) return PS_ERR_INVALID;
        r.count = int(items);
        ctas += (items + G - 1) / G;
        const size_t M = size_t(1) << c.logM;
        smem = std::max(smem, size_t(G) * (M + M / 8 + (size_t(1) << r.logT)) * sizeof(double2));
      }
    }
    if (L.n == 0) continue;
    if (ctas > 0x7fffffff) return PS_ERR_INVALID;
    const int rc = go(L, nt, int(ctas), smem);
    if (rc != PS_OK) return rc;
  }
  return PS_OK;
}

static RingPart ring_part(const double2* phase, const double* map, int nf, int pack) {
  return {pack ? (nf + 1) / 2 : nf, pack, nf, const_cast<double2*>(phase), const_cast<double*>(map)};
}

static int ring_synth(const Plan& P, const RingClassList* cls, int ncls, const RingPart* part, int nparts,
                      double2* minus, int64_t map_stride, cudaStream_t st) {
  auto go = [&](const RingLaunch& L, int nt, int ctas, size_t smem) -> int {
    const auto kern = minus ? (nt == 512 ? ring_synth_f64<512, true> : ring_synth_f64<256, true>)
                            : (nt == 512 ? ring_synth_f64<512, false> : ring_synth_f64<256, false>);
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return PS_ERR_CUDA;
    StatScope sc(PS_K_FFT_SYNTH, 0.0, 0.0, st);
    kern<<<ctas, nt, smem, st>>>(L, minus);
    PS_LAUNCH_CHECK();
    return PS_OK;
  };
  return ring_launches(P, cls, ncls, map_stride, part, nparts, go);
}

static int ring_adjoint(const Plan& P, const RingClassList* cls, int ncls, const RingPart* part, int nparts,
                        const double2* minus, int64_t map_stride, cudaStream_t st) {
  auto go = [&](const RingLaunch& L, int nt, int ctas, size_t smem) -> int {
    const auto kern = minus ? (nt == 512 ? ring_adjoint_f64<512, true> : ring_adjoint_f64<256, true>)
                            : (nt == 512 ? ring_adjoint_f64<512, false> : ring_adjoint_f64<256, false>);
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return PS_ERR_CUDA;
    StatScope sc(PS_K_FFT_ADJOINT, 0.0, 0.0, st);
    kern<<<ctas, nt, smem, st>>>(L, minus);
    PS_LAUNCH_CHECK();
    return PS_OK;
  };
  return ring_launches(P, cls, ncls, map_stride, part, nparts, go);
}

int launch_ring_synth_f64(const Plan& P, const RingClassList* cls, int ncls, const double2* phase, double* map,
                          double2* minus, int64_t map_stride, int nf, int pack, cudaStream_t st) {
  const RingPart part = ring_part(phase, map, nf, pack);
  return ring_synth(P, cls, ncls, &part, 1, minus, map_stride, st);
}

int launch_ring_adjoint_f64(const Plan& P, const RingClassList* cls, int ncls, const double* map,
                            const double2* minus, int64_t map_stride, double2* phase, int nf, int pack, cudaStream_t st) {
  const RingPart part = ring_part(phase, map, nf, pack);
  return ring_adjoint(P, cls, ncls, &part, 1, minus, map_stride, st);
}

// T at map and (Q, U) in the two components after it, of `batch` maps; phases of the two spins apart.
int launch_ring_synth_fields_f64(const Plan& P, const RingClassList* cls, int ncls, const double2* phase0,
                                 const double2* phase2, double* map, int64_t map_stride, int batch, cudaStream_t st) {
  const RingPart part[2] = {ring_part(phase0, map, batch, 0), ring_part(phase2, map + P.npix, 2 * batch, 1)};
  return ring_synth(P, cls, ncls, part, 2, nullptr, map_stride, st);
}

int launch_ring_adjoint_fields_f64(const Plan& P, const RingClassList* cls, int ncls, const double* map,
                                   int64_t map_stride, double2* phase0, double2* phase2, int batch, cudaStream_t st) {
  const RingPart part[2] = {ring_part(phase0, map, batch, 0), ring_part(phase2, map + P.npix, 2 * batch, 1)};
  return ring_adjoint(P, cls, ncls, part, 2, nullptr, map_stride, st);
}

}  // namespace ps
