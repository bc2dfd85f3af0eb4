// alm [B][ncomp][nalm] (maps `stride` apart) -> almT [nalm][B][ncomp], the B operand order of the mixed-precision
// Legendre stages, optionally times a factor per (component, lm).
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
                                                const double* __restrict__ lscale, double2* __restrict__ almT, int nf,
                                                int ncomp, int64_t nalm, int nt, int lt) {
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
        double2 v = alm[b * stride + c * nalm + i0 + j];
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

}  // namespace

int launch_alm_to_T(const double2* alm, int64_t stride, const double* lscale, double2* almT, int B, int ncomp,
                    int64_t nalm, cudaStream_t st) {
  const int nf = B * ncomp;
  StatScope sc(PS_K_LAYOUT, 0.0, 32.0 * nf * double(nalm), st);
  const int gy = (nf + 31) / 32, nt = (nf + gy - 1) / gy;
  int lt = 5;
  while (lt < 9 && (nt << (lt + 1)) <= SLOTS) ++lt;
  const dim3 grid(unsigned((nalm + (1 << lt) - 1) >> lt), gy < 65535 ? gy : 65535);
  alm_to_T<<<grid, 256, 0, st>>>(alm, stride, lscale, almT, nf, ncomp, nalm, nt, lt);
  PS_LAUNCH_CHECK();
  return PS_OK;
}

}  // namespace ps
