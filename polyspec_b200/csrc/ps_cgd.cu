// One step of the single-map CG (polyspec/weighting.py:326-339) besides its transforms, three launches with the
// scalars left on the device:
//   ps_cgd_apply:     q = beam y + C^-1 p (in place over y, y the transformed part of A p) and p^T q
//   ps_cgd_update:    alpha = rz / p^T q; x += alpha p, r -= alpha q; z = Sigma r, r^T z and beta (harmonic
//                     preconditioner), or without z
//   ps_cgd_rz:        r^T z and beta, of a z computed elsewhere
//   ps_cgd_direction: p = z + beta p and beam p, the next transform's input
//
// A vector has (1 or 3) (lmax+1)(lmax+2)/2 values, at lmax 256 1.6 MB: in cache, and the launches are what a step costs.
// A block per 256 (l, m) keeps the chip busy at that size; the blocks leave their share of the inner product in
// memory and the one that finishes last adds the shares up, in their order, so that no launch and no wait on the
// host follows.  As elementwise, einsum (a batched matrix-vector library call of 34 us each) and reduction calls the
// same part of a step took 28 launches and 160 us of kernels for T, E, B at lmax 256, with these kernels 25 us.
#include "ps_common.cuh"
#include "ps_stats.cuh"

namespace ps {
namespace {

constexpr int CGD_THREADS = 256, CGD_MAX_BLOCKS = 1024;
enum { RZ = 0, PQ = 1, BETA = 2, NO_STEP = 3 };  // scalars of the solve

// r^T z or p^T A p is zero: there is no alpha or beta, and the vectors stay as they are.
__device__ __forceinline__ bool no_step(const double* scal) {
  return __ldcg(scal + RZ) == 0.0 || __ldcg(scal + PQ) == 0.0;
}

// Sum of the blocks' v by the last of them to arrive, on its thread 0; other threads get false.
__device__ bool last_block_sum(double v, double* partial, unsigned* counter, double& total) {
  __shared__ double sw[CGD_THREADS / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto block_sum = [&](double t) {  // on thread 0
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
    if (lane == 0) sw[warp] = t;
    __syncthreads();
    t = 0.0;
    if (threadIdx.x == 0)
      for (int k = 0; k < CGD_THREADS / 32; ++k) t += sw[k];
    return t;
  };
  v = block_sum(v);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = v;
    __threadfence();
    last = atomicInc(counter, gridDim.x - 1) == gridDim.x - 1;  // back to 0 with the last block
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double t = 0.0;
  for (int i = threadIdx.x; i < int(gridDim.x); i += CGD_THREADS) t += __ldcg(partial + i);
  total = block_sum(t);
  return threadIdx.x == 0;
}

__device__ __forceinline__ double re_dot(double2 a, double2 b) { return a.x * b.x + a.y * b.y; }

template <int NF>
__device__ __forceinline__ double2 row_times(const double* __restrict__ S, int a, const double2 (&v)[NF], int64_t nalm,
                                             int64_t i) {
  double2 s = make_double2(0.0, 0.0);
#pragma unroll
  for (int b = 0; b < NF; ++b) s = cfma(__ldg(S + (int64_t(a) * NF + b) * nalm + i), v[b], s);
  return s;
}

template <int NF>
__global__ void __launch_bounds__(CGD_THREADS) cgd_apply(const double* __restrict__ S, const double* __restrict__ beam,
                                                         const double* __restrict__ w, const double2* __restrict__ p,
                                                         double2* __restrict__ y, int64_t nalm, double* scal,
                                                         double* partial, unsigned* counter) {
  double dot = 0.0;
  for (int64_t i = int64_t(blockIdx.x) * CGD_THREADS + threadIdx.x; i < nalm; i += int64_t(gridDim.x) * CGD_THREADS) {
    double2 v[NF];
    double d = 0.0;
#pragma unroll
    for (int a = 0; a < NF; ++a) v[a] = p[a * nalm + i];
#pragma unroll
    for (int a = 0; a < NF; ++a) {
      const double2 q = cfma(beam[a * nalm + i], y[a * nalm + i], row_times<NF>(S, a, v, nalm, i));
      y[a * nalm + i] = q;
      d += re_dot(v[a], q);
    }
    dot = fma(w[i], d, dot);
  }
  double total;
  if (last_block_sum(dot, partial, counter, total)) scal[PQ] = total;
}

// every block has read rz before the last one replaces it
__device__ __forceinline__ void next_rz(double total, double* scal) {
  scal[NO_STEP] = 0.0;
  scal[BETA] = total / scal[RZ];
  scal[RZ] = total;
}

template <int NF, bool SIGMA>
__global__ void __launch_bounds__(CGD_THREADS) cgd_update(const double* __restrict__ S, const double* __restrict__ w,
                                                          const double2* __restrict__ p, const double2* __restrict__ q,
                                                          double2* __restrict__ x, double2* __restrict__ r,
                                                          double2* __restrict__ z, int64_t nalm, double* scal,
                                                          double* partial, unsigned* counter) {
  if (no_step(scal)) {
    if (SIGMA && blockIdx.x == 0 && threadIdx.x == 0) scal[NO_STEP] = 1.0;
    return;
  }
  const double alpha = __ldcg(scal + RZ) / __ldcg(scal + PQ);
  double dot = 0.0;
  for (int64_t i = int64_t(blockIdx.x) * CGD_THREADS + threadIdx.x; i < nalm; i += int64_t(gridDim.x) * CGD_THREADS) {
    double2 v[NF];
#pragma unroll
    for (int a = 0; a < NF; ++a) {
      x[a * nalm + i] = cfma(alpha, p[a * nalm + i], x[a * nalm + i]);
      v[a] = cfma(-alpha, q[a * nalm + i], r[a * nalm + i]);
      r[a * nalm + i] = v[a];
    }
    if constexpr (SIGMA) {
      double d = 0.0;
#pragma unroll
      for (int a = 0; a < NF; ++a) {
        const double2 s = row_times<NF>(S, a, v, nalm, i);
        z[a * nalm + i] = s;
        d += re_dot(v[a], s);
      }
      dot = fma(w[i], d, dot);
    }
  }
  if constexpr (SIGMA) {
    double total;
    if (last_block_sum(dot, partial, counter, total)) next_rz(total, scal);
  }
}

template <int NF>
__global__ void __launch_bounds__(CGD_THREADS) cgd_rz(const double* __restrict__ w, const double2* __restrict__ r,
                                                      const double2* __restrict__ z, int64_t nalm, double* scal,
                                                      double* partial, unsigned* counter) {
  if (no_step(scal)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) scal[NO_STEP] = 1.0;
    return;
  }
  double dot = 0.0;
  for (int64_t i = int64_t(blockIdx.x) * CGD_THREADS + threadIdx.x; i < nalm; i += int64_t(gridDim.x) * CGD_THREADS) {
    double d = 0.0;
#pragma unroll
    for (int a = 0; a < NF; ++a) d += re_dot(r[a * nalm + i], z[a * nalm + i]);
    dot = fma(w[i], d, dot);
  }
  double total;
  if (last_block_sum(dot, partial, counter, total)) next_rz(total, scal);
}

__global__ void __launch_bounds__(CGD_THREADS) cgd_direction(const double* __restrict__ beam,
                                                             const double2* __restrict__ z, double2* __restrict__ p,
                                                             double2* __restrict__ bp, int64_t n,
                                                             const double* __restrict__ scal) {
  if (scal[NO_STEP] != 0.0) return;
  const double beta = scal[BETA];
  for (int64_t i = int64_t(blockIdx.x) * CGD_THREADS + threadIdx.x; i < n; i += int64_t(gridDim.x) * CGD_THREADS) {
    const double2 v = cfma(beta, p[i], z[i]);
    p[i] = v;
    bp[i] = cscale(v, beam[i]);
  }
}

int cgd_blocks(int64_t n) {
  const int64_t b = (n + CGD_THREADS - 1) / CGD_THREADS;
  return int(b < CGD_MAX_BLOCKS ? b : CGD_MAX_BLOCKS);
}

}  // namespace
}  // namespace ps

using namespace ps;

// workspace: the arrival counter (zero before the first call, and left zero), then the blocks' shares
static unsigned* cgd_counter(void* ws) { return static_cast<unsigned*>(ws); }
static double* cgd_partial(void* ws) { return static_cast<double*>(ws) + 1; }
static const double2* c2(const double* p) { return reinterpret_cast<const double2*>(p); }
static double2* c2(double* p) { return reinterpret_cast<double2*>(p); }

extern "C" int ps_cgd_workspace_bytes(size_t* bytes) {
  if (!bytes) return PS_ERR_INVALID;
  *bytes = sizeof(double) * (1 + CGD_MAX_BLOCKS);
  return PS_OK;
}

extern "C" int ps_cgd_apply(const double* S, const double* beam, const double* w, const double* p, double* y, int nf,
                            int64_t nalm, double* scal, void* workspace, size_t workspace_bytes, cudaStream_t stream) {
  if (!S || !beam || !w || !p || !y || !scal || p == y || (nf != 1 && nf != 3) || nalm <= 0) return PS_ERR_INVALID;
  if (!workspace || workspace_bytes < sizeof(double) * (1 + CGD_MAX_BLOCKS)) return PS_ERR_WORKSPACE;
  StatScope sc(PS_K_VECTOR, 16.0 * nf * nf * nalm, (48.0 * nf + 8.0 * nf * nf) * nalm, stream);
  const auto kern = nf == 1 ? cgd_apply<1> : cgd_apply<3>;
  kern<<<cgd_blocks(nalm), CGD_THREADS, 0, stream>>>(S, beam, w, c2(p), c2(y), nalm, scal, cgd_partial(workspace),
                                                     cgd_counter(workspace));
  PS_LAUNCH_CHECK();
  return PS_OK;
}

extern "C" int ps_cgd_update(const double* Sigma, const double* w, const double* p, const double* q, double* x,
                             double* r, double* z, int nf, int64_t nalm, double* scal, void* workspace,
                             size_t workspace_bytes, cudaStream_t stream) {
  if (!w || !p || !q || !x || !r || !scal || (Sigma && !z) || (nf != 1 && nf != 3) || nalm <= 0) return PS_ERR_INVALID;
  if (!workspace || workspace_bytes < sizeof(double) * (1 + CGD_MAX_BLOCKS)) return PS_ERR_WORKSPACE;
  StatScope sc(PS_K_VECTOR, 16.0 * nf * nf * nalm, (112.0 * nf + 8.0 * nf * nf) * nalm, stream);
  const auto kern = Sigma ? (nf == 1 ? cgd_update<1, true> : cgd_update<3, true>)
                          : (nf == 1 ? cgd_update<1, false> : cgd_update<3, false>);
  kern<<<cgd_blocks(nalm), CGD_THREADS, 0, stream>>>(Sigma, w, c2(p), c2(q), c2(x), c2(r), c2(z), nalm, scal,
                                                     cgd_partial(workspace), cgd_counter(workspace));
  PS_LAUNCH_CHECK();
  return PS_OK;
}

extern "C" int ps_cgd_rz(const double* w, const double* r, const double* z, int nf, int64_t nalm, double* scal,
                         void* workspace, size_t workspace_bytes, cudaStream_t stream) {
  if (!w || !r || !z || !scal || (nf != 1 && nf != 3) || nalm <= 0) return PS_ERR_INVALID;
  if (!workspace || workspace_bytes < sizeof(double) * (1 + CGD_MAX_BLOCKS)) return PS_ERR_WORKSPACE;
  StatScope sc(PS_K_VECTOR, 5.0 * nf * nalm, 32.0 * nf * nalm, stream);
  const auto kern = nf == 1 ? cgd_rz<1> : cgd_rz<3>;
  kern<<<cgd_blocks(nalm), CGD_THREADS, 0, stream>>>(w, c2(r), c2(z), nalm, scal, cgd_partial(workspace),
                                                     cgd_counter(workspace));
  PS_LAUNCH_CHECK();
  return PS_OK;
}

extern "C" int ps_cgd_direction(const double* beam, const double* z, double* p, double* beam_p, int nf, int64_t nalm,
                                const double* scal, cudaStream_t stream) {
  if (!beam || !z || !p || !beam_p || !scal || (nf != 1 && nf != 3) || nalm <= 0) return PS_ERR_INVALID;
  StatScope sc(PS_K_VECTOR, 6.0 * nf * nalm, 72.0 * nf * nalm, stream);
  cgd_direction<<<cgd_blocks(nf * nalm), CGD_THREADS, 0, stream>>>(beam, c2(z), c2(p), c2(beam_p), nf * nalm, scal);
  PS_LAUNCH_CHECK();
  return PS_OK;
}
