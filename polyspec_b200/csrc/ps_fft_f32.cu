// FP32 ring transforms of the mixed-precision HEALPix SHT (maps stay FP64 in
// HBM; the per-ring phases and the FFTs run in FP32).  Per ring of nphi pixels:
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
// One launch takes the rings of every work length up to 8192 (a second one 16384): a CTA of
// 512 threads runs G = 512 / T transforms of one length class, T = length / 16, neighbouring
// fields first.  Phases are stored map-innermost ([ring][m][field], as the Legendre GEMMs read
// and write them): the synthesis folds them into shared memory, and the adjoint writes them from
// there, with the G fields of one (ring, m) in neighbouring lanes, so that whole 32-byte sectors
// move (a transform's own threads would use 8 bytes of each).
//
// A transform is a sequence of radix-2 stages with twiddles from tables, three (first pass: up to
// four) at a time in registers between shared-memory exchanges (one element of padding per 16):
// Stockham order for power-of-two rings, Bluestein's chirp-z convolution of power-of-two length
// M >= 2 nphi - 1 for the others (decimation in frequency, spectrum, decimation in time), whose
// zero upper half of the input and unused upper half of the output are skipped and whose middle
// passes and product stay in registers.  The ring rotations e^{i m phi0}, the chirps, the spectra
// and the twiddles (level after level, contiguous) are tables of the plan computed in FP64.
#include <algorithm>

#include "ps_common.cuh"
#include "ps_stats.cuh"

namespace ps {

__device__ __forceinline__ float2 fadd2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 fsub2(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// Complex products with the contraction written out, so that a transform's bits do not depend on how the compiler
// groups the stages: the two forms differ in which product of the imaginary part is rounded.
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y)));
}
__device__ __forceinline__ float2 fmul2x(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 fconj2(float2 a) { return make_float2(a.x, -a.y); }

__host__ __device__ constexpr int frev(int k, int bits) {
  int r = 0;
  for (int b = 0; b < bits; ++b) r |= ((k >> b) & 1) << (bits - 1 - b);
  return r;
}
__host__ __device__ constexpr int flog2(int n) { return n <= 1 ? 0 : 1 + flog2(n / 2); }
__device__ __forceinline__ int fpad(int i) { return i + (i >> 4); }

// twiddle e^{-2 pi i j / 2^s}, j < 2^(s-1): level s starts at 2^(s-1) - 1 of the plan's table
__device__ __forceinline__ float2 twf(const float2* __restrict__ tw, int s, int j) {
  return __ldg(&tw[(1 << (s - 1)) - 1 + j]);
}

// log2 R radix-2 stages of decimation in frequency on the points j + k q, k < R, of a block of 2^s = R q points:
// natural order in, position k holds the points of frequency rev(k) mod R out.  HALF: x[R/2..] are zero (not read).
// AT: number of stages of the transform before these (mod 3); every third stage uses fmul2, the others fmul2x.
template <int R, int AT, bool HALF = false>
__device__ __forceinline__ void dif_stages(float2* x, const float2* __restrict__ tw, int s, int j, int q) {
#pragma unroll
  for (int len = R; len > 1; len /= 2, --s) {
    const bool first = (flog2(R) - flog2(len) + AT) % 3 == 0;
#pragma unroll
    for (int k = 0; k < len / 2; ++k) {
      const float2 w = twf(tw, s, j + k * q);
#pragma unroll
      for (int b = 0; b < R; b += len) {
        if (HALF && len == R) {
          x[k + R / 2] = first ? fmul2(x[k], w) : fmul2x(x[k], w);
        } else {
          const float2 d = fsub2(x[b + k], x[b + k + len / 2]);
          x[b + k] = fadd2(x[b + k], x[b + k + len / 2]);
          x[b + k + len / 2] = first ? fmul2(d, w) : fmul2x(d, w);
        }
      }
    }
  }
}
// The inverse stages (decimation in time): position k holds frequency rev(k) in, natural order out.
template <int R>
__device__ __forceinline__ void dit_stages(float2* x, const float2* __restrict__ tw, int s, int j, int q) {
  s -= flog2(R) - 1;
#pragma unroll
  for (int len = 2; len <= R; len *= 2, ++s) {
#pragma unroll
    for (int k = 0; k < len / 2; ++k) {
      const float2 w = fconj2(twf(tw, s, j + k * q));
#pragma unroll
      for (int b = 0; b < R; b += len) {
        const float2 v = fmul2(x[b + k + len / 2], w);
        x[b + k + len / 2] = fsub2(x[b + k], v);
        x[b + k] = fadd2(x[b + k], v);
      }
    }
  }
}

// Bluestein convolution in place: in.load<H>(x, t, q) gives the inputs at t + k q, k < H (times the chirp, zero from N
// on; they may be a's own elements), out(j, v), j < N <= M/2, takes the results.  M = R1 8^n, n >= 1.
template <int R1, class In, class Out>
__device__ __forceinline__ void bluestein_f(float2* a, int N, int M, int logM, const float2* __restrict__ spec,
                                            const float2* __restrict__ tw, int u, int T, const In& in,
                                            const Out& out) {
  constexpr int H = R1 / 2, LR = flog2(R1);
  const int q1 = M / R1;
  for (int t = u; t < q1; t += T) {
    float2 x[R1];
    in.template load<H>(x, t, q1);
    dif_stages<R1, 0, true>(x, tw, logM, t, q1);
#pragma unroll
    for (int k = 0; k < R1; ++k) a[fpad(t + k * q1)] = x[k];
  }
  __syncthreads();
  int s = logM - LR;  // log2 of the block length
  for (; s > 3; s -= 3) {
    const int lq = s - 3, q = 1 << lq;
    for (int t = u; t < M / 8; t += T) {
      const int j = t & (q - 1), i0 = ((t >> lq) << s) + j;
      float2 x[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = a[fpad(i0 + k * q)];
      dif_stages<8, LR % 3>(x, tw, s, j, q);
#pragma unroll
      for (int k = 0; k < 8; ++k) a[fpad(i0 + k * q)] = x[k];
    }
    __syncthreads();
  }
  for (int t = u; t < M / 8; t += T) {
    float2 x[8];
    const float4* sp = reinterpret_cast<const float4*>(spec) + 4 * t;  // a spectrum starts at a multiple of 32 elements
    float4 b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) b[k] = __ldg(&sp[k]);
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = a[fpad(8 * t + k)];
    dif_stages<8, LR % 3>(x, tw, 3, 0, 1);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      x[k] = fmul2(x[k], (k & 1) ? make_float2(b[k / 2].z, b[k / 2].w) : make_float2(b[k / 2].x, b[k / 2].y));
    dit_stages<8>(x, tw, 3, 0, 1);
#pragma unroll
    for (int k = 0; k < 8; ++k) a[fpad(8 * t + k)] = x[k];
  }
  __syncthreads();
  for (s = 6; s <= logM - LR; s += 3) {
    const int lq = s - 3, q = 1 << lq;
    for (int t = u; t < M / 8; t += T) {
      const int j = t & (q - 1), i0 = ((t >> lq) << s) + j;
      float2 x[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = a[fpad(i0 + k * q)];
      dit_stages<8>(x, tw, s, j, q);
#pragma unroll
      for (int k = 0; k < 8; ++k) a[fpad(i0 + k * q)] = x[k];
    }
    __syncthreads();
  }
  for (int t = u; t < q1; t += T) {
    float2 x[R1];
#pragma unroll
    for (int k = 0; k < R1; ++k) x[k] = a[fpad(t + k * q1)];
    dit_stages<R1>(x, tw, logM, t, q1);
#pragma unroll
    for (int k = 0; k < H; ++k)
      if (t + k * q1 < N) out(t + k * q1, x[k]);
  }
}

// Stockham DFT of length M = R1 8^n, T >= M / 16.  LOCAL: in reads a's own elements.  out is called by the thread that
// read a's elements of the same indices last.
template <int R1, bool LOCAL, class In, class Out>
__device__ __forceinline__ void stockham_f(float2* a, int M, int logM, const float2* __restrict__ tw, int u, int T,
                                           const In& in, const Out& out) {
  constexpr int LR = flog2(R1), NB = 16 / R1;
  const int q1 = M / R1;
  {
    float2 x[NB][R1];
#pragma unroll
    for (int h = 0; h < NB; ++h)
      if (u + h * T < q1) in.template load<R1>(x[h], u + h * T, q1);
    if (LOCAL) __syncthreads();
#pragma unroll
    for (int h = 0; h < NB; ++h) {
      const int t = u + h * T;
      if (t >= q1) continue;
      dif_stages<R1, 0>(x[h], tw, logM, t, q1);
      if (logM == LR) {
#pragma unroll
        for (int k = 0; k < R1; ++k) out(frev(k, LR), x[h][k]);
      } else {
#pragma unroll
        for (int k = 0; k < R1; ++k) a[fpad(t * R1 + frev(k, LR))] = x[h][k];
      }
    }
  }
  const int q = M / 8;
  for (int ln = LR; ln < logM; ln += 3) {
    __syncthreads();
    const bool last = ln + 3 == logM;
    float2 x[2][8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = u + h * T;
      if (t >= q) continue;
#pragma unroll
      for (int k = 0; k < 8; ++k) x[h][k] = a[fpad(t + k * q)];
      dif_stages<8, LR % 3>(x[h], tw, logM - ln, t >> ln, 1 << (logM - ln - 3));
      if (last) {
#pragma unroll
        for (int k = 0; k < 8; ++k) out(t + frev(k, 3) * q, x[h][k]);
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
      for (int k = 0; k < 8; ++k) a[fpad(i0 + (frev(k, 3) << ln))] = x[h][k];
    }
  }
}

template <bool LOCAL, class In, class Out>
__device__ __forceinline__ void ring_dft_f(bool blue, float2* a, int N, int M, int logM,
                                           const float2* __restrict__ spec, const float2* __restrict__ tw, int u, int T,
                                           const In& in, const Out& out) {
  const int r = logM % 3;  // the same for all transforms of a CTA
  if (blue) {
    if (r == 0) bluestein_f<8>(a, N, M, logM, spec, tw, u, T, in, out);
    else if (r == 1) bluestein_f<16>(a, N, M, logM, spec, tw, u, T, in, out);
    else bluestein_f<4>(a, N, M, logM, spec, tw, u, T, in, out);
  } else {
    if (r == 0) stockham_f<8, LOCAL>(a, M, logM, tw, u, T, in, out);
    else if (r == 1) stockham_f<16, LOCAL>(a, M, logM, tw, u, T, in, out);
    else stockham_f<4, LOCAL>(a, M, logM, tw, u, T, in, out);
  }
}

// ------------------------------------------------------------------ kernels
// One length class of a launch: CTAs [cta0, next class's cta0) run its `count` items, G to a CTA.
struct RingClassF {
  int cta0, count, logM, logT, blue;
  const int* rings;
};
constexpr int RING_CLASSES_F = 28, RING_NT = 512;
struct RingLaunchF {
  int n, units, pack, mmax, R;
  int64_t nf, npix, map_stride;  // map_stride: from one map to the next
  const RingInfo* rings;
  const float2 *tw, *spec, *rot, *chirp;
  const int64_t *spec_off, *chirp_off;
  RingClassF c[RING_CLASSES_F];
};

// item -> (ring, unit) -> the two packed rows of phases and pixels
struct RingItemF {
  int N;
  bool va, vb;
  const float2* rot;
  const float2 *chirp, *spec;
  int64_t pa, pb, pix_a, pix_b, start_a, start_b;  // first phases; first pixels of the two rows, and in their maps
};
struct RingCtaF {  // what the transforms of a CTA share
  int M, logM, logT, T, G, item0, count, blue;
  const int* rings;
};
__device__ __forceinline__ RingCtaF ring_cta_f(const RingLaunchF& L) {
  int ci = 0;
  while (ci + 1 < L.n && int(blockIdx.x) >= L.c[ci + 1].cta0) ++ci;
  const RingClassF& c = L.c[ci];
  RingCtaF r;
  r.logM = c.logM;
  r.M = 1 << c.logM;
  r.logT = c.logT;
  r.T = 1 << c.logT;
  r.G = RING_NT >> c.logT;
  r.item0 = (int(blockIdx.x) - c.cta0) * r.G;
  r.count = c.count;
  r.blue = c.blue;
  r.rings = c.rings;
  return r;
}
__device__ __forceinline__ RingItemF ring_item_f(const RingLaunchF& L, const RingCtaF& c, int grp) {
  RingItemF it;
  const int item = c.item0 + grp;
  it.va = item < c.count;
  const int ring = it.va ? item / L.units : 0, unit = it.va ? item - ring * L.units : 0;
  const int ira = c.rings[ring], irb = L.pack ? ira : L.R - 1 - ira;
  const RingInfo g = L.rings[ira];
  it.N = g.nphi;
  it.start_a = g.start;
  it.start_b = L.rings[irb].start;
  it.pix_a = unit * L.map_stride + it.start_a;
  it.pix_b = unit * L.map_stride + (L.pack ? L.npix : 0) + it.start_b;
  it.vb = it.va && (L.pack || irb != ira);
  const int64_t row = int64_t(L.mmax + 1) * L.nf;
  it.pa = ira * row + (L.pack ? 2 * unit : unit);
  it.pb = irb * row + (L.pack ? 2 * unit + 1 : unit);
  it.rot = L.rot + int64_t(min(ira, L.R - 1 - ira)) * (L.mmax + 1);  // e^{i m phi0} of this ring
  it.chirp = c.blue ? L.chirp + L.chirp_off[g.bs_slot] : nullptr;
  it.spec = c.blue ? L.spec + L.spec_off[g.bs_slot] : nullptr;
  return it;
}
__device__ __forceinline__ size_t ring_smem_f(const RingCtaF& c) { return size_t(c.M + (c.M >> 4)); }

// Folded phases of the CTA's transforms into shared memory: conj(c_a) + i conj(c_b) (times the chirp) with
// c_k = sum_{m = k mod N} F_m e^{i m phi0} + sum_{m = -k mod N, m > 0} conj(...), zero from N to the end of what the
// first pass reads.
__device__ __forceinline__ void fold_phases(const RingLaunchF& L, const RingCtaF& c, const float2* __restrict__ phase,
                                            float2* smem) {
  const int g = threadIdx.x & (c.G - 1), mmax = L.mmax;
  const RingItemF it = ring_item_f(L, c, g);
  float2* a = smem + g * ring_smem_f(c);
  const int N = it.N, top = c.blue ? c.M / 2 : c.M;
  const int64_t nf = L.nf;
  const float2* pha = phase + it.pa;
  const float2* phb = phase + it.pb;
  for (int kk = threadIdx.x >> (9 - c.logT); kk < top; kk += c.T) {
    float2 v = make_float2(0.f, 0.f);
    if (kk < N) {
      float2 ca = make_float2(0.f, 0.f), cb = ca;
      if (it.va) {
        for (int m = kk; m <= mmax; m += N) {
          const float2 e = it.rot[m];
          ca = fadd2(ca, fmul2x(pha[int64_t(m) * nf], e));
          if (it.vb) cb = fadd2(cb, fmul2x(phb[int64_t(m) * nf], e));
        }
        for (int m = (kk == 0) ? N : N - kk; m <= mmax; m += N) {
          const float2 e = it.rot[m];
          ca = fadd2(ca, fconj2(fmul2x(pha[int64_t(m) * nf], e)));
          if (it.vb) cb = fadd2(cb, fconj2(fmul2x(phb[int64_t(m) * nf], e)));
        }
      }
      // a real field keeps only Re(c_0) (F_0's imaginary part drops out of the
      // real map); it must not leak into the partner field of the packed pair
      if (kk == 0) { ca.y = 0.f; cb.y = 0.f; }
      v = make_float2(ca.x + cb.y, -ca.y + cb.x);  // conj(ca) + i conj(cb)
      if (c.blue) v = fmul2(v, it.chirp[kk]);
    }
    a[fpad(kk)] = v;
  }
}

// The CTA's transforms, natural order in shared memory, to phases.
__device__ __forceinline__ void store_phases(const RingLaunchF& L, const RingCtaF& c, const float2* smem,
                                             float2* __restrict__ phase) {
  const int g = threadIdx.x & (c.G - 1);
  const RingItemF it = ring_item_f(L, c, g);
  if (!it.va) return;
  const float2* a = smem + g * ring_smem_f(c);
  const int N = it.N;
  const int64_t nf = L.nf;
  for (int m = threadIdx.x >> (9 - c.logT); m <= L.mmax; m += c.T) {
    const int k = m < N ? m : m % N;
    const float2 z = a[fpad(k)], z2 = fconj2(a[fpad(k == 0 ? 0 : N - k)]);
    const float2 e = fconj2(it.rot[m]);
    const float2 xa = make_float2(0.5f * (z.x + z2.x), 0.5f * (z.y + z2.y));
    // (z - z2) / (2i) = -i (z - z2) / 2
    const float2 xb = make_float2(0.5f * (z.y - z2.y), -0.5f * (z.x - z2.x));
    phase[it.pa + int64_t(m) * nf] = fmul2(xa, e);
    if (it.vb) phase[it.pb + int64_t(m) * nf] = fmul2(xb, e);
  }
}

struct LocalIn {  // the transform's own elements, folded before
  const float2* a;
  template <int K>
  __device__ __forceinline__ void load(float2* x, int t, int q) const {
#pragma unroll
    for (int i = 0; i < K; ++i) x[i] = a[fpad(t + i * q)];
  }
};

__device__ __forceinline__ float2 dechirp(float2 y, const float2* __restrict__ chirp, int j, float s) {
  const float2 v = fmul2(y, chirp[j]);
  return make_float2(v.x * s, v.y * s);
}

// synthesis: phase [R][mmax+1][nf] (complex64) -> maps (float64), or (PAIR, packed) complex maps Q + iU at map and
// Q - iU at minus (complex128)
template <bool PAIR>
__global__ void __launch_bounds__(RING_NT, 2) ring_synth_f32(const __grid_constant__ RingLaunchF L,
                                                             const float2* __restrict__ phase,
                                                             double* __restrict__ map, double2* __restrict__ minus) {
  extern __shared__ float2 fbuf[];
  const RingCtaF c = ring_cta_f(L);
  fold_phases(L, c, phase, fbuf);
  __syncthreads();
  const int grp = threadIdx.x >> c.logT, u = threadIdx.x & (c.T - 1);
  const RingItemF it = ring_item_f(L, c, grp);
  float2* a = fbuf + grp * ring_smem_f(c);
  double* oa = map + it.pix_a;
  double* ob = map + it.pix_b;
  double2* op = reinterpret_cast<double2*>(map) + it.pix_a;
  double2* om = minus + it.pix_a;
  const float inv = 1.0f / float(c.M);
  auto out = [&](int j, float2 y) {
    if (c.blue) y = dechirp(y, it.chirp, j, inv);
    if constexpr (PAIR) {
      if (it.va) {
        op[j] = make_double2(y.x, y.y);
        om[j] = make_double2(y.x, -y.y);
      }
    } else {
      if (it.va) oa[j] = double(y.x);
      if (it.vb) ob[j] = double(y.y);
    }
  };
  ring_dft_f<true>(c.blue, a, it.N, c.M, c.logM, it.spec, L.tw, u, c.T, LocalIn{a}, out);
}

template <bool PAIR>
struct MapIn {
  const double *ia, *ib;
  const double2 *ip, *im;
  const float2* chirp;
  int N;
  bool va, vb, blue;
  template <int K>
  __device__ __forceinline__ void load(float2* x, int t, int q) const {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int j = t + i * q;
      if constexpr (PAIR) {
        const double2 z = make_double2(0.0, 0.0), p = va && j < N ? ip[j] : z, n = va && j < N ? im[j] : z;
        x[i] = make_float2(float(0.5 * (p.x + n.x)), float(0.5 * (p.y - n.y)));
      } else {
        x[i] = make_float2(va && j < N ? float(ia[j]) : 0.f, vb && j < N ? float(ib[j]) : 0.f);
      }
    }
    if (blue) {
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (t + i * q < N) x[i] = fmul2(x[i], chirp[t + i * q]);
    }
  }
};

// adjoint: maps (float64), or (PAIR, packed) Q = Re (p + n) / 2, U = Im (p - n) / 2 of the complex maps p and
// n = minus -> phase [R][mmax+1][nf] (complex64)
template <bool PAIR>
__global__ void __launch_bounds__(RING_NT, 2) ring_adjoint_f32(const __grid_constant__ RingLaunchF L,
                                                               const double* __restrict__ map,
                                                               const double2* __restrict__ minus,
                                                               float2* __restrict__ phase) {
  extern __shared__ float2 fbuf[];
  const RingCtaF c = ring_cta_f(L);
  const int grp = threadIdx.x >> c.logT, u = threadIdx.x & (c.T - 1);
  const RingItemF it = ring_item_f(L, c, grp);
  float2* a = fbuf + grp * ring_smem_f(c);
  const MapIn<PAIR> in{map + it.pix_a, map + it.pix_b, reinterpret_cast<const double2*>(map) + it.pix_a,
                       minus + it.pix_a, it.chirp, it.N, it.va, it.vb, c.blue != 0};
  const float inv = 1.0f / float(c.M);
  auto out = [&](int k, float2 y) { a[fpad(k)] = c.blue ? dechirp(y, it.chirp, k, inv) : y; };
  ring_dft_f<false>(c.blue, a, it.N, c.M, c.logM, it.spec, L.tw, u, c.T, in, out);
  __syncthreads();
  store_phases(L, c, fbuf, phase);
}

// synthesis -> pixel weights -> adjoint of the same rings, in place on the phases:
//   phase [R][mmax+1][nf] (complex64)  ->  P'_m = sum_j w_j map_j e^{-i m (phi0 + 2 pi j / nphi)}
// with map = the ring's synthesis of the phases and w the per-pixel weight of each field
// (weight [ncw][npix]: field a reads component 0, field b component 1 for a spin map, or
// component 0 on the mirror ring for spin 0).  The map never leaves shared memory.  A CTA reads
// every phase it writes before the first barrier, so in place is safe.
__global__ void __launch_bounds__(RING_NT, 2) ring_roundtrip_f32(const __grid_constant__ RingLaunchF L,
                                                                 const double* __restrict__ weight,
                                                                 float2* __restrict__ phase) {
  extern __shared__ float2 fbuf[];
  const RingCtaF c = ring_cta_f(L);
  fold_phases(L, c, phase, fbuf);
  __syncthreads();
  const int grp = threadIdx.x >> c.logT, u = threadIdx.x & (c.T - 1);
  const RingItemF it = ring_item_f(L, c, grp);
  float2* a = fbuf + grp * ring_smem_f(c);
  const double* wa = weight + it.start_a;
  const double* wb = weight + (L.pack ? L.npix : 0) + it.start_b;
  const float inv = 1.0f / float(c.M);
  auto weighted = [&](int j, float2 y) {
    if (c.blue) y = dechirp(y, it.chirp, j, inv);
    y = make_float2(it.va ? float(wa[j]) * y.x : 0.f, it.vb ? float(wb[j]) * y.y : 0.f);
    a[fpad(j)] = c.blue ? fmul2(y, it.chirp[j]) : y;  // the input of the second transform
  };
  ring_dft_f<true>(c.blue, a, it.N, c.M, c.logM, it.spec, L.tw, u, c.T, LocalIn{a}, weighted);
  __syncthreads();
  if (c.blue) {  // the convolution left its tail from N on
    for (int j = it.N + u; j < c.M / 2; j += c.T) a[fpad(j)] = make_float2(0.f, 0.f);
    __syncthreads();
  }
  auto out = [&](int k, float2 y) { a[fpad(k)] = c.blue ? dechirp(y, it.chirp, k, inv) : y; };
  ring_dft_f<true>(c.blue, a, it.N, c.M, c.logM, it.spec, L.tw, u, c.T, LocalIn{a}, out);
  __syncthreads();
  store_phases(L, c, fbuf, phase);
}

// ------------------------------------------------------------------ launch
template <class Launch>
static int ring_launches_f(const Plan& P, const RingClassList* cls, int ncls, int64_t map_stride, int nf, int pack,
                           Launch go) {
  RingLaunchF L;
  L.units = pack ? (nf + 1) / 2 : nf;
  L.pack = pack; L.nf = nf; L.mmax = P.mmax; L.R = P.R; L.npix = P.npix; L.map_stride = map_stride; L.rings = P.d_rings;
  L.tw = P.d_twiddle_f; L.spec = P.d_bs_spec_f; L.spec_off = P.d_bs_off;
  L.rot = P.d_rot_f; L.chirp = P.d_chirp_f; L.chirp_off = P.d_chirp_off;
  for (int big = 1; big >= 0; --big) {  // work length 16384 first, then all others, longest first
    size_t smem = 0;
    int64_t ctas = 0;
    double share = 0.0;
    L.n = 0;
    for (int i = 0; i < ncls; ++i) {
      const RingClassList& c = cls[i];
      const int count = pack ? c.count : c.count_n;
      if ((c.logM > 13) != (big == 1) || count == 0) continue;
      if (L.n == RING_CLASSES_F) return PS_ERR_UNSUPPORTED;
      RingClassF& r = L.c[L.n++];
      r.cta0 = int(ctas);
      r.logM = c.logM;
      r.logT = std::max(5, std::min(9, c.logM - 4));
      r.blue = c.blue;
      r.rings = pack ? c.rings : c.rings_n;
      const int64_t items = int64_t(count) * L.units, G = RING_NT >> r.logT;
      if (items > 0x7fffffff) return PS_ERR_INVALID;
      r.count = int(items);
      ctas += (items + G - 1) / G;
      share += double(count);
      const size_t M = size_t(1) << c.logM;
      smem = std::max(smem, size_t(G) * (M + M / 16) * sizeof(float2));
    }
    if (L.n == 0) continue;
    if (ctas > 0x7fffffff) return PS_ERR_INVALID;
    const int rc = go(L, int(ctas), smem, share / double(P.R));
    if (rc != PS_OK) return rc;
  }
  return PS_OK;
}

template <class K>
static bool ring_smem_ok(K kern, size_t smem) {
  return smem <= 48 * 1024 ||
         cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess;
}

int launch_ring_synth_f32(const Plan& P, const RingClassList* cls, int ncls, const float2* phase, double* map,
                          double2* minus, int64_t map_stride, int nf, int pack, cudaStream_t st) {
  auto go = [&](const RingLaunchF& L, int ctas, size_t smem, double) -> int {
    const auto kern = minus ? ring_synth_f32<true> : ring_synth_f32<false>;
    if (!ring_smem_ok(kern, smem)) return PS_ERR_CUDA;
    StatScope sc(PS_K_FFT_SYNTH, 0.0, 0.0, st);
    kern<<<ctas, RING_NT, smem, st>>>(L, phase, map, minus);
    PS_LAUNCH_CHECK();
    return PS_OK;
  };
  return ring_launches_f(P, cls, ncls, map_stride, nf, pack, go);
}

int launch_ring_adjoint_f32(const Plan& P, const RingClassList* cls, int ncls, const double* map,
                            const double2* minus, int64_t map_stride, float2* phase, int nf, int pack, cudaStream_t st) {
  auto go = [&](const RingLaunchF& L, int ctas, size_t smem, double) -> int {
    const auto kern = minus ? ring_adjoint_f32<true> : ring_adjoint_f32<false>;
    if (!ring_smem_ok(kern, smem)) return PS_ERR_CUDA;
    StatScope sc(PS_K_FFT_ADJOINT, 0.0, 0.0, st);
    kern<<<ctas, RING_NT, smem, st>>>(L, map, minus, phase);
    PS_LAUNCH_CHECK();
    return PS_OK;
  };
  return ring_launches_f(P, cls, ncls, map_stride, nf, pack, go);
}

int launch_ring_roundtrip_f32(const Plan& P, const RingClassList* cls, int ncls, float2* phase, const double* weight,
                              int nf, int pack, cudaStream_t st) {
  // the pixel weights and the phases, read and written once
  const double bytes = double(P.npix) * 8.0 * (pack ? 2.0 : 1.0) + 2.0 * 8.0 * P.R * (P.mmax + 1) * nf;
  auto go = [&](const RingLaunchF& L, int ctas, size_t smem, double share) -> int {
    if (!ring_smem_ok(ring_roundtrip_f32, smem)) return PS_ERR_CUDA;
    StatScope sc(PS_K_FFT_SYNTH, 0.0, bytes * share, st);
    ring_roundtrip_f32<<<ctas, RING_NT, smem, st>>>(L, weight, phase);
    PS_LAUNCH_CHECK();
    return PS_OK;
  };
  return ring_launches_f(P, cls, ncls, 0, nf, pack, go);
}

}  // namespace ps
