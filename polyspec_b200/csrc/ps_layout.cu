// alm [B][ncomp][nalm] (maps `stride` apart) -> almT [nalm][B][ncomp], the B operand order of the mixed-precision
// Legendre stages, optionally times a factor per (component, lm); grad: from alm [B][nalm], (G, C) = (-alm, 0).
//
// Bound by HBM (16 bytes read and written per value).  A tile of up to 32 fields x up to 512 values goes through shared
// memory, so that both sides move in long runs; one thread per output value, with two 64-bit divisions and reads
// 16 nalm bytes apart, took 116 us for the 33 + 66 fields of a T, E, B batch at lmax 511 (64 us at the copy rate), the
// tile takes 90 us.  The fields are split evenly over the tiles and the tile is as long as they leave room for.
#include "ps_common.cuh"
#include "ps_stats.cuh"

namespace ps {
namespace {

constexpr int SLOTS = 1024;  // values per tile

// tile: nt fields x 2^lt values, nt << lt <= SLOTS
__global__ void __launch_bounds__(256) alm_to_T(const double2* __restrict__ alm, int64_t stride,
                                                const double* __restrict__ lscale, bool grad,
                                                double2* __restrict__ almT, int nf, int ncomp, int64_t nalm, int nt,
                                                int lt) {
  __shared__ double2 s[SLOTS + 32];  // rows of 2^lt + 1
  const int tl = 1 << lt;
  const int64_t i0 = int64_t(blockIdx.x) << lt;
  const int n = int(min(int64_t(tl), nalm - i0));
  for (int f0 = blockIdx.y * nt; f0 < nf; f0 += gridDim.y * nt) {
    const int nr = min(nt, nf - f0);
#pragma unroll
    for (int k = 0; k < SLOTS / 256; ++k) {
      const int t = threadIdx.x + 256 * k, r = t >> lt, j = t & (tl - 1);
      if (r < nr && j < n) {
        const int f = f0 + r, b = f / ncomp, c = f - b * ncomp;
        double2 v = grad && c ? make_double2(0.0, 0.0) : alm[b * stride + c * nalm + i0 + j];
        if (grad && !c) v = make_double2(-v.x, -v.y);
        if (lscale) v = cscale(v, lscale[c * nalm + i0 + j]);
        s[r * (tl + 1) + j] = v;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SLOTS / 256; ++k) {
      const int t = threadIdx.x + 256 * k, j = t / nr, r = t - j * nr;
      if (j < n) almT[(i0 + j) * nf + f0 + r] = s[r * (tl + 1) + j];
    }
    __syncthreads();
  }
}

// (G, C) [B][2][nalm] -> plus = -(G + iC), minus = -(-1)^s (G - iC), each [B][nalm]
__global__ void __launch_bounds__(256) gc_to_pm(const double2* __restrict__ gc, double2* __restrict__ plus,
                                                double2* __restrict__ minus, int64_t nalm, double sign) {
  const int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x;
  if (i >= nalm) return;
  const int64_t b = blockIdx.y;
  const double2 G = gc[2 * b * nalm + i], C = gc[(2 * b + 1) * nalm + i];
  plus[b * nalm + i] = make_double2(C.y - G.x, -G.y - C.x);
  minus[b * nalm + i] = make_double2(sign * (G.x + C.y), sign * (G.y - C.x));
}

}  // namespace

int launch_gc_to_pm(const double2* gc, double2* plus, double2* minus, int B, int64_t nalm, int spin, cudaStream_t st) {
  StatScope sc(PS_K_LAYOUT, 0.0, 64.0 * B * double(nalm), st);
  for (int b = 0; b < B; b += 65535) {
    const int64_t o = b * nalm;
    gc_to_pm<<<dim3(unsigned((nalm + 255) / 256), B - b < 65535 ? B - b : 65535), 256, 0, st>>>(
        gc + 2 * o, plus + o, minus + o, nalm, (spin & 1) ? 1.0 : -1.0);
    PS_LAUNCH_CHECK();
  }
  return PS_OK;
}

int launch_alm_to_T(const double2* alm, int64_t stride, const double* lscale, bool grad, double2* almT, int B, int ncomp,
                    int64_t nalm, cudaStream_t st) {
  const int nf = B * ncomp;
  StatScope sc(PS_K_LAYOUT, 0.0, 32.0 * nf * double(nalm), st);
  const int gy = (nf + 31) / 32, nt = (nf + gy - 1) / gy;
  int lt = 5;
  while (lt < 9 && (nt << (lt + 1)) <= SLOTS) ++lt;
  const dim3 grid(unsigned((nalm + (1 << lt) - 1) >> lt), gy < 65535 ? gy : 65535);
  alm_to_T<<<grid, 256, 0, st>>>(alm, stride, lscale, grad, almT, nf, ncomp, nalm, nt, lt);
  PS_LAUNCH_CHECK();
  return PS_OK;
}

}  // namespace ps
