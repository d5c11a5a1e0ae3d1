// Krylov vector kernels and diagnostics reductions (FP64).
// Reductions are deterministic: a fixed grid of RED_BLOCKS blocks with a fixed
// element-to-thread map writes per-block partials, and a second pass sums the
// partials in a fixed order, so a result never depends on scheduling.
// They replace the deal.II vector operations used by SolverCG/SolverGMRES and
// the diagnostics of Atmospheric_Flow.cc:991-1087, 1140-1148.
#include <cfloat>
#include <cmath>

#include "atm_device.cuh"

namespace atm {

namespace {
constexpr int RT = 256;  // threads per reduction block
constexpr int MAXM = 32;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}
// op: 0 sum, 1 max, 2 min; result valid in thread 0
template <int OP>
__device__ double block_reduce(double v, double *sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = OP == 0 ? warp_sum(v) : (OP == 1 ? warp_max(v) : warp_min(v));
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  if (wid == 0) {
    v = lane < nw ? sh[lane] : (OP == 0 ? 0.0 : (OP == 1 ? -DBL_MAX : DBL_MAX));
    v = OP == 0 ? warp_sum(v) : (OP == 1 ? warp_max(v) : warp_min(v));
  }
  return v;
}

__global__ void k_copy(double *__restrict__ d, const double *__restrict__ s, long n) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    d[i] = s[i];
}
__global__ void k_fill(double *__restrict__ d, double v, long n) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    d[i] = v;
}
__global__ void k_axpy(double *__restrict__ y, double a, const double *__restrict__ x, long n) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] += a * x[i];
}
__global__ void k_xmy_scaled(double *__restrict__ d, const double *__restrict__ dg,
                             const double *__restrict__ b, const double *__restrict__ t, long n) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    d[i] = dg[i] * (b[i] - t[i]);
}
__global__ void k_scale_inv_norm(double *__restrict__ d, const double *__restrict__ s,
                                 const double *__restrict__ nsq, long n) {
  // one root and division per block: per thread they cost more FP64 time than
  // the vector takes to move
  __shared__ double inv;
  if (threadIdx.x == 0) inv = 1.0 / sqrt(*nsq);
  __syncthreads();
  const double a = inv;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    d[i] = s[i] * a;
}

__global__ void k_dot_partial(const double *__restrict__ x, const double *__restrict__ y, long n,
                              double *__restrict__ red) {
  __shared__ double sh[RT / 32];
  double acc = 0.0;
  for (long i = (long)blockIdx.x * RT + threadIdx.x; i < n; i += (long)RED_BLOCKS * RT)
    acc = fma(x[i], y[i], acc);
  acc = block_reduce<0>(acc, sh);
  if (threadIdx.x == 0) red[blockIdx.x] = acc;
}

// out[row] = sum of red[row*RED_BLOCKS .. +RED_BLOCKS) (OP 0), max (1), min (2)
template <int OP>
__global__ void k_finalize(const double *__restrict__ red, double *__restrict__ out) {
  __shared__ double sh[RT / 32];
  const double *r = red + (long)blockIdx.x * RED_BLOCKS;
  double acc = OP == 0 ? 0.0 : (OP == 1 ? -DBL_MAX : DBL_MAX);
  for (int i = threadIdx.x; i < RED_BLOCKS; i += RT)
    acc = OP == 0 ? acc + r[i] : (OP == 1 ? fmax(acc, r[i]) : fmin(acc, r[i]));
  acc = block_reduce<OP>(acc, sh);
  if (threadIdx.x == 0) out[blockIdx.x] = acc;
}

__global__ void k_multiaxpy(double *__restrict__ w, const double *__restrict__ V, long ldv,
                            int m, const double *__restrict__ h, double sign, long n) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int l = 0; l < m; ++l) s = fma(h[l], V[l * ldv + i], s);
    w[i] += sign * s;
  }
}

// ------------------------------------------------------ Arnoldi sweeps --
// One sweep over the basis V_0..V_{M-1} and the new direction w:
//   MODE 0: out_l = V_l . w
//   MODE 1: w -= sum_l h_l V_l, then out_l = V_l . w
//   MODE 2: w -= sum_l h_l V_l, then out_0 = w . w
// Block (b, s) works on its share of segment s (the whole vector, or one
// member's range eoff[s]..eoff[s+1]); h and out are [row][segment].  All M dot
// products stay in registers, so V is read once per sweep, and M is a template
// parameter so that an element's M loads are in flight together.
//
// Bound by FP64 instructions at small vectors (n = 320,000: 28 vectors fit L2):
// reducing M sums over a warp value by value takes 5 M additions per warp, as
// much as the elements of a short thread.  The warp instead halves the set of
// values it carries at each exchange (31 additions for 32 sums), and a thread
// takes at least four elements.  The last block of a segment to finish sums the
// partials in block order, which needs no second launch and never depends on
// scheduling.  In MODE 2 it also writes all coefficients to the pinned
// mirror `host` (rows 0.. h1, 32.. h2, 64 |w|^2), which saves the copy.
// At n = 320,000, m = 8 / 20: 12 / 28 us (MODE 0), 17 / 34 us (MODE 1); before,
// a kernel per eight vectors and one for the sum took 25-41 us each.
template <int M, int MODE>
__global__ void __launch_bounds__(RT, 1)
    k_arnoldi(double *__restrict__ w, const double *__restrict__ V, long ldv,
              const double *__restrict__ h, const long *__restrict__ eoff, long n,
              double *__restrict__ red, double *__restrict__ out, unsigned *__restrict__ ticket,
              const double *__restrict__ h1, double *__restrict__ host) {
  constexpr int NS = MODE == 2 ? 1 : M;  // sums, and the power of two above
  constexpr int NV = NS <= 1 ? 1 : NS <= 2 ? 2 : NS <= 4 ? 4 : NS <= 8 ? 8 : NS <= 16 ? 16 : 32;
  __shared__ double sh[NV][RT / 32];
  __shared__ bool last;
  const int seg = blockIdx.y, ns = gridDim.y, b = blockIdx.x, nb = gridDim.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long lo = eoff ? eoff[seg] : 0, hi = eoff ? eoff[seg + 1] : n;
  double hc[MODE ? M : 1], acc[NV];
#pragma unroll
  for (int l = 0; l < NV; ++l) acc[l] = 0.0;
  if (MODE) {
#pragma unroll
    for (int l = 0; l < M; ++l) hc[MODE ? l : 0] = h[(long)l * ns + seg];
  }
  for (long i = lo + (long)b * RT + threadIdx.x; i < hi; i += (long)nb * RT) {
    double v[M], wi = w[i];
#pragma unroll
    for (int l = 0; l < M; ++l) v[l] = V[l * ldv + i];
    if (MODE) {
      double s = 0.0;
#pragma unroll
      for (int l = 0; l < M; ++l) s = fma(hc[MODE ? l : 0], v[l], s);
      wi -= s;
      w[i] = wi;
    }
    if (MODE == 2) {
      acc[0] = fma(wi, wi, acc[0]);
    } else {
#pragma unroll
      for (int l = 0; l < NS; ++l) acc[l] = fma(v[l], wi, acc[l]);
    }
  }
  // after the exchanges the lane holds the sum of value lane / (32 / NV)
  int s = NV;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    if (s > 1) {
      const bool up = lane & off;
#pragma unroll
      for (int l = 0; l < NV / 2; ++l)
        if (l < s / 2) {
          const double give = up ? acc[l] : acc[l + s / 2], keep = up ? acc[l + s / 2] : acc[l];
          acc[l] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
      s /= 2;
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
    }
  }
  if (lane % (32 / NV) == 0) sh[lane / (32 / NV)][wid] = acc[0];
  __syncthreads();
  double *part = red + (long)seg * 32 * nb;
  if (threadIdx.x < NS) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < RT / 32; ++k) t += sh[threadIdx.x][k];
    part[(long)threadIdx.x * nb + b] = t;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket + seg, 1u) == (unsigned)nb - 1;
  __syncthreads();
  if (!last) return;
  for (int l = wid; l < NS; l += RT / 32) {
    double t = 0.0;
    for (int k = lane; k < nb; k += 32) t += __ldcg(part + (long)l * nb + k);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
    if (lane == 0) {
      out[(long)l * ns + seg] = t;
      if (MODE == 2) host[64L * ns + seg] = t;
    }
  }
  if (MODE == 2)
    for (int l = threadIdx.x; l < M; l += RT) {
      host[(long)l * ns + seg] = h1[(long)l * ns + seg];
      host[(32L + l) * ns + seg] = h[(long)l * ns + seg];
    }
  if (threadIdx.x == 0) ticket[seg] = 0;
}

template <int MODE>
void arnoldi_sweep(cudaStream_t st, dim3 grid, double *w, const double *V, long n, int m,
                   const double *h, const long *eoff, double *red, double *out, unsigned *ticket,
                   const double *h1, double *host) {
  switch (m) {
#define ARNOLDI_M(M)                                                                        \
  case M:                                                                                   \
    k_arnoldi<M, MODE><<<grid, RT, 0, st>>>(w, V, n, h, eoff, n, red, out, ticket, h1, host); \
    break;
#define ARNOLDI_M4(M) ARNOLDI_M(M) ARNOLDI_M(M + 1) ARNOLDI_M(M + 2) ARNOLDI_M(M + 3)
    ARNOLDI_M4(1) ARNOLDI_M4(5) ARNOLDI_M4(9) ARNOLDI_M4(13)
    ARNOLDI_M4(17) ARNOLDI_M4(21) ARNOLDI_M4(25) ARNOLDI_M4(29)
#undef ARNOLDI_M4
#undef ARNOLDI_M
  }
  g_kernel_launches.fetch_add(1);
}

__global__ void k_maxdiff_partial(const double *__restrict__ a, const double *__restrict__ b,
                                  long n, double *__restrict__ red) {
  __shared__ double sh[RT / 32];
  double m0 = 0.0, m1 = 0.0;
  for (long i = (long)blockIdx.x * RT + threadIdx.x; i < n; i += (long)RED_BLOCKS * RT) {
    const double ai = a[i];
    m1 = fmax(m1, fabs(ai));
    m0 = fmax(m0, fabs(b ? ai - b[i] : ai));
  }
  m0 = block_reduce<1>(m0, sh);
  if (threadIdx.x == 0) red[blockIdx.x] = m0;
  m1 = block_reduce<1>(m1, sh);
  if (threadIdx.x == 0) red[RED_BLOCKS + blockIdx.x] = m1;
}

__global__ void k_diag_partial(const double *__restrict__ rho, const double *__restrict__ u,
                               const double *__restrict__ p, int nc, int nn2,
                               double *__restrict__ red) {
  __shared__ double sh[RT / 32];
  double rmin = DBL_MAX, rmax = 0.0, cmax = 0.0, umax = 0.0;
  const long n = (long)nc * nn2;
  for (long i = (long)blockIdx.x * RT + threadIdx.x; i < n; i += (long)RED_BLOCKS * RT) {
    const long c = i / nn2, j = i - c * nn2;
    const double r = rho[i];
    rmin = fmin(rmin, r);
    rmax = fmax(rmax, fabs(r));
    cmax = fmax(cmax, sqrt(GAS_GAMMA * p[i] / r));
    const double u0 = u[(c * 2) * nn2 + j], u1 = u[(c * 2 + 1) * nn2 + j];
    umax = fmax(umax, sqrt(u0 * u0 + u1 * u1));
  }
  double v = block_reduce<2>(rmin, sh);
  if (threadIdx.x == 0) red[blockIdx.x] = v;
  v = block_reduce<1>(rmax, sh);
  if (threadIdx.x == 0) red[RED_BLOCKS + blockIdx.x] = v;
  v = block_reduce<1>(cmax, sh);
  if (threadIdx.x == 0) red[2 * RED_BLOCKS + blockIdx.x] = v;
  v = block_reduce<1>(umax, sh);
  if (threadIdx.x == 0) red[3 * RED_BLOCKS + blockIdx.x] = v;
}

// relax u toward (ub0, ub1), or toward the per-node target velocity (same
// layout as u) when one is given
__global__ void k_sponge(double *__restrict__ u, const double *__restrict__ alpha, double dt,
                         double ub0, double ub1, const double *__restrict__ target,
                         const double *__restrict__ dts, int nc, int nn2) {
  const long n = (long)nc * nn2;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const long c = i / nn2, j = i - c * nn2;
    const double a = dt * (dts ? dts[c] : 1.0) * alpha[i];
    if (a == 0.0) continue;
    const long i0 = (c * 2) * nn2 + j, i1 = (c * 2 + 1) * nn2 + j;
    const double t0 = target ? target[i0] : ub0, t1 = target ? target[i1] : ub1;
    u[i0] = (u[i0] + a * t0) / (1.0 + a);
    u[i1] = (u[i1] + a * t1) / (1.0 + a);
  }
}

inline int grid_for(long n) {
  long g = (n + 255) / 256;
  if (g > 152L * 16) g = 152L * 16;  // grid-stride beyond 16 blocks per SM
  return (int)(g < 1 ? 1 : g);
}
}  // namespace

int vec_copy(cudaStream_t st, double *dst, const double *src, long n) {
  if (n <= 0 || dst == src) return ATM_OK;
  k_copy<<<grid_for(n), 256, 0, st>>>(dst, src, n);
  ATM_CHECK_LAUNCH("k_copy");
  return ATM_OK;
}
int vec_fill(cudaStream_t st, double *dst, double v, long n) {
  if (n <= 0) return ATM_OK;
  k_fill<<<grid_for(n), 256, 0, st>>>(dst, v, n);
  ATM_CHECK_LAUNCH("k_fill");
  return ATM_OK;
}
int vec_axpy(cudaStream_t st, double *y, double a, const double *x, long n) {
  if (n <= 0) return ATM_OK;
  k_axpy<<<grid_for(n), 256, 0, st>>>(y, a, x, n);
  ATM_CHECK_LAUNCH("k_axpy");
  return ATM_OK;
}
int vec_xmy_scaled(cudaStream_t st, double *dst, const double *d, const double *b,
                   const double *t, long n) {
  k_xmy_scaled<<<grid_for(n), 256, 0, st>>>(dst, d, b, t, n);
  ATM_CHECK_LAUNCH("k_xmy_scaled");
  return ATM_OK;
}
int vec_scale_by_inv_norm(cudaStream_t st, double *dst, const double *src, const double *nsq,
                          long n) {
  k_scale_inv_norm<<<grid_for(n), 256, 0, st>>>(dst, src, nsq, n);
  ATM_CHECK_LAUNCH("k_scale_inv_norm");
  return ATM_OK;
}
int vec_dot(cudaStream_t st, const double *x, const double *y, long n, double *red,
            double *out) {
  k_dot_partial<<<RED_BLOCKS, RT, 0, st>>>(x, y, n, red);
  k_finalize<0><<<1, RT, 0, st>>>(red, out);
  ATM_CHECK_LAUNCH("vec_dot");
  return ATM_OK;
}
int vec_multiaxpy(cudaStream_t st, double *w, const double *V, long ldv, int m,
                  const double *h, double sign, long n) {
  if (m < 1) return ATM_OK;
  k_multiaxpy<<<grid_for(n), 256, 0, st>>>(w, V, ldv, m, h, sign, n);
  ATM_CHECK_LAUNCH("k_multiaxpy");
  return ATM_OK;
}
int arnoldi_blocks(long n, int m, int segments) {
  // at least four elements per thread; one block per SM where the kernel's
  // registers (m > 8) leave room for one, two otherwise
  const long most = (m > 8 ? 152L : 304L) / (segments < 1 ? 1 : segments);
  long g = n / (4L * RT * (segments < 1 ? 1 : segments));
  if (g > most) g = most;
  return (int)(g < 1 ? 1 : g);
}
int arnoldi_sweeps(cudaStream_t st, double *V, long n, int j, double *w, const long *eoff,
                   int segments, double *red, double *coef, unsigned *ticket, double *host) {
  const int m = j + 1;
  if (m > MAXM) {
    set_error("Arnoldi step: more basis vectors than the reduction buffer holds");
    return ATM_BAD_ARG;
  }
  double *h1 = coef, *h2 = coef + 32L * segments, *nsq = coef + 64L * segments;
  const dim3 grid(arnoldi_blocks(n, m, segments), segments);
  arnoldi_sweep<0>(st, grid, w, V, n, m, nullptr, eoff, red, h1, ticket, nullptr, nullptr);
  ATM_CUDA(cudaGetLastError());
  arnoldi_sweep<1>(st, grid, w, V, n, m, h1, eoff, red, h2, ticket, nullptr, nullptr);
  ATM_CUDA(cudaGetLastError());
  arnoldi_sweep<2>(st, grid, w, V, n, m, h2, eoff, red, nsq, ticket, h1, host);
  ATM_CUDA(cudaGetLastError());
  return ATM_OK;
}
int arnoldi_step(cudaStream_t st, double *V, long n, int j, double *w, double *red,
                 double *dsmall, double *h_pinned, double *hcol, double *hn) {
  int rc;
  if ((rc = arnoldi_sweeps(st, V, n, j, w, nullptr, 1, red, dsmall,
                           reinterpret_cast<unsigned *>(dsmall + 248), h_pinned)))
    return rc;
  // scaled while the host waits; a zero or non-finite norm ends the cycle and
  // nobody reads V_{j+1}
  if ((rc = vec_scale_by_inv_norm(st, V + (long)(j + 1) * n, w, dsmall + 64, n))) return rc;
  ATM_CUDA(cudaStreamSynchronize(st));
  for (int l = 0; l <= j; ++l) hcol[l] = h_pinned[l] + h_pinned[32 + l];
  *hn = std::sqrt(h_pinned[64]);
  return ATM_OK;
}
int vec_maxdiff(cudaStream_t st, const double *a, const double *b, long n, double *red,
                double *out) {
  k_maxdiff_partial<<<RED_BLOCKS, RT, 0, st>>>(a, b, n, red);
  k_finalize<1><<<2, RT, 0, st>>>(red, out);
  ATM_CHECK_LAUNCH("vec_maxdiff");
  return ATM_OK;
}
int vec_diagnostics(cudaStream_t st, const double *rho, const double *u, const double *p,
                    int nc, int nn2, double *red, double *out) {
  k_diag_partial<<<RED_BLOCKS, RT, 0, st>>>(rho, u, p, nc, nn2, red);
  k_finalize<2><<<1, RT, 0, st>>>(red, out);
  k_finalize<1><<<3, RT, 0, st>>>(red + RED_BLOCKS, out + 1);
  ATM_CHECK_LAUNCH("vec_diagnostics");
  return ATM_OK;
}
int vec_sponge(cudaStream_t st, double *u, const double *alpha, double dt, double ub0,
               double ub1, const double *target, const double *dts, int nc, int nn2) {
  const long n = (long)nc * nn2;
  k_sponge<<<grid_for(n), 256, 0, st>>>(u, alpha, dt, ub0, ub1, target, dts, nc, nn2);
  ATM_CHECK_LAUNCH("k_sponge");
  return ATM_OK;
}

}  // namespace atm

// ------------------------------------------------------------------------
// FMA throughput probe: 8 independent FMA chains per thread on a grid of
// 8 blocks per SM; used to measure the FP64 / FP32 denominators of the
// compute roofline on the machine the bench runs on.
namespace atm {
namespace {
template <typename T>
__global__ void k_fma_probe(T *out, int iters, T a, T b) {
  T x0 = (T)threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3;
  T x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
  for (int i = 0; i < iters; ++i) {
    x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
    x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
  }
  out[blockIdx.x * blockDim.x + threadIdx.x] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}
template <typename T>
int probe(int iters, double *gflops) {
  int dev = 0, nsm = 0;
  ATM_CUDA(cudaGetDevice(&dev));
  ATM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int blocks = nsm * 8, threads = 256;
  T *out = nullptr;
  ATM_CUDA(cudaMalloc(&out, sizeof(T) * blocks * threads));
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  k_fma_probe<T><<<blocks, threads>>>(out, 16, (T)0.999, (T)0.001);
  cudaEventRecord(e0);
  k_fma_probe<T><<<blocks, threads>>>(out, iters, (T)0.999, (T)0.001);
  cudaEventRecord(e1);
  cudaError_t err = cudaEventSynchronize(e1);
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  g_kernel_launches.fetch_add(2);
  if (err != cudaSuccess) return cuda_fail(err, "fma probe");
  *gflops = 2.0 * 8.0 * iters * (double)blocks * threads / (ms * 1e-3) / 1e9;
  return ATM_OK;
}
}  // namespace
}  // namespace atm

extern "C" int atm_probe_fma_peak(double *fp64_gflops, double *fp32_gflops) {
  if (!fp64_gflops || !fp32_gflops) return ATM_BAD_ARG;
  int rc = atm::probe<double>(4000, fp64_gflops);
  if (rc) return rc;
  return atm::probe<float>(100000, fp32_gflops);
}
