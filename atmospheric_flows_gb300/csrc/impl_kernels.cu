// Implicit-block kernels (FP64):
//   B   pressure gradient, p -> velocity   euler_operator.h:1512-1617
//   C   enthalpy divergence, w -> pressure euler_operator.h:1413-1507
//   D   internal-energy mass               euler_operator.h:1386-1408
//   A   rho_fix-weighted velocity mass     euler_operator.h:2330-2357
//   rho mass                               euler_operator.h:717-740
//   inverse diagonals                      euler_operator.h:2458-2626
// plus the exact cell-wise inverses of the (weighted) DG mass matrices.
// Because every mass-type block of this DG discretisation is cell-local,
// A^{-1}, M^{-1} and D^{-1} are applied exactly with one dense (k+1)^2 block
// per cell instead of the reference's CG iterations (euler_operator.h:2391-2397,
// Atmospheric_Flow.cc:452-536); the Schur apply S p = D p - C A^{-1} B p is
// then two fused kernels: (B, A^{-1}) and (C, D, Jacobi).
#include "schur_kernels.cuh"

namespace atm {

int upload_basis_impl(const double *t) { return upload_basis_here(t); }

// hanging-face instantiations of B and C/D live in hang_schur.cu (FP64) and
// hang_schur_f.cu (FP32 multigrid levels)
int launch_B_hang(const atm_ctx &c, double *dst, const double *p, double coeff, int mode);
int launch_CD_hang(const atm_ctx &c, double *dst, const double *w, const double *p,
                   double coeff, int mode);
template <typename T>
int level_B_hang(const OpView<T> &o, T *dst, const T *p, T cB, int mode);
template <typename T>
int level_CD_hang(const OpView<T> &o, T *dst, const T *w, const T *p, T cC, int mode,
                  const ChebArgs<T> *ch);
// general_schur_f.cu (FP32 levels, conforming)
int general_B_f(const OpView<float> &o, float *dst, const float *p, float cB);
int general_CD_f(const OpView<float> &o, float *dst, const float *w, const float *p, float cC,
                 int mode, const ChebArgs<float> *ch);

// ============================================================ mass apply ===
// dst = M_w src for NCOMP components; weight tile (rho) or constant scale
template <int K, int NCOMP, bool WEIGHTED, typename T>
__global__ void __launch_bounds__(Cfg<K>::THREADS)
    k_mass(T *__restrict__ dst, const T *__restrict__ src,
           const T *__restrict__ weight, T scale, MeshT<T> mesh) {
  using C = Cfg<K>;
  constexpr int NN = C::NN, NQ = C::NQ, NN2 = C::NN2, NQ2 = C::NQ2, CPB = C::CPB;
  constexpr int NT = NCOMP + (WEIGHTED ? 1 : 0);
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T *sm = reinterpret_cast<T *>(sm_raw);
  T *tiles = sm;
  T *xab = tiles + CPB * NT * NN2;  // [CPB][NCOMP][NN*NQ]
  const int tid = threadIdx.x, lc = tid / NQ, col = tid - lc * NQ;
  const int c0 = blockIdx.x * CPB;
  const int cnt = min(CPB, mesh.nc - c0);
  load_tiles<K>(tiles, NT, 0, src, NCOMP, c0, cnt);
  if (WEIGHTED) load_tiles<K>(tiles, NT, NCOMP, weight, 1, c0, cnt);
  __syncthreads();
  const bool active = lc < cnt;
  const int c = c0 + lc;
  T Sx[NN], Dx[NN];
  load_rows<K>(col, Sx, Dx);
  if (active) {
    const T *tl = tiles + lc * NT * NN2;
    T wv[NQ];
    if (WEIGHTED) eval_col<K>(tl + NCOMP * NN2, Sx, wv);
    const T *G = mesh.jw + c * mesh.jw_stride;
#pragma unroll
    for (int comp = 0; comp < NCOMP; ++comp) {
      T v[NQ], V[NQ];
      eval_col<K>(tl + comp * NN2, Sx, v);
#pragma unroll
      for (int qz = 0; qz < NQ; ++qz) {
        const T jxw = G[qz * NQ + col];
        V[qz] = (WEIGHTED ? wv[qz] * v[qz] : scale * v[qz]) * jxw;
      }
      integrate_col_z<K, true, false>(V, V, V, xab + (lc * NCOMP + comp) * NN * NQ, (T *)nullptr,
                                      col);
    }
  }
  __syncthreads();
  if (active && col < NN) {
    T St[NQ], Dt[NQ];
    load_cols<K>(col, St, Dt);
#pragma unroll
    for (int comp = 0; comp < NCOMP; ++comp) {
      T out[NN];
      integrate_out<K, false>(xab + (lc * NCOMP + comp) * NN * NQ, (const T *)nullptr, St, Dt, out);
      T *d = dst + ((long)c * NCOMP + comp) * NN2;
#pragma unroll
      for (int iz = 0; iz < NN; ++iz) d[iz * NN + col] = out[iz];
    }
  }
}

// ===================================================== inverse diagonal ===
template <int K, bool WEIGHTED, typename T>
__global__ void __launch_bounds__(Cfg<K>::THREADS)
    k_invdiag(T *__restrict__ out, int ncomp, const T *__restrict__ weight,
              T scale, MeshT<T> mesh) {
  using C = Cfg<K>;
  constexpr int NN = C::NN, NQ = C::NQ, NN2 = C::NN2, NQ2 = C::NQ2, CPB = C::CPB;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T *sm = reinterpret_cast<T *>(sm_raw);
  T *tiles = sm;                      // [CPB][NN2] weight
  T *xab = tiles + CPB * NN2;         // [CPB][NN*NQ]
  const int tid = threadIdx.x, lc = tid / NQ, col = tid - lc * NQ;
  const int c0 = blockIdx.x * CPB;
  const int cnt = min(CPB, mesh.nc - c0);
  if (WEIGHTED) load_tiles<K>(tiles, 1, 0, weight, 1, c0, cnt);
  __syncthreads();
  const bool active = lc < cnt;
  const int c = c0 + lc;
  T Sx[NN], Dx[NN];
  load_rows<K>(col, Sx, Dx);
  if (active) {
    T wv[NQ];
    if (WEIGHTED) eval_col<K>(tiles + lc * NN2, Sx, wv);
    const T *G = mesh.jw + c * mesh.jw_stride;
#pragma unroll
    for (int iz = 0; iz < NN; ++iz) {
      T s = T(0.0);
#pragma unroll
      for (int qz = 0; qz < NQ; ++qz) {
        const T b = bS<K, T>(qz, iz);
        const T wj = (WEIGHTED ? wv[qz] : scale) * G[qz * NQ + col];
        s = fma(b * b, wj, s);
      }
      xab[lc * NN * NQ + iz * NQ + col] = s;
    }
  }
  __syncthreads();
  if (active && col < NN) {
#pragma unroll
    for (int iz = 0; iz < NN; ++iz) {
      T s = T(0.0);
#pragma unroll
      for (int qx = 0; qx < NQ; ++qx) {
        const T b = bS<K, T>(qx, col);
        s = fma(b * b, xab[lc * NN * NQ + iz * NQ + qx], s);
      }
      const T inv = T(1.0) / s;
      for (int comp = 0; comp < ncomp; ++comp)
        out[((long)c * ncomp + comp) * NN2 + iz * NN + col] = inv;
    }
  }
}

// ================================================= exact block inverse ===
// G lanes per cell (32 / G cells per warp).  The (weighted) cell mass matrix
//   M[(iz,ix),(jz,jx)] = sum_q S(qz,iz)S(qz,jz) S(qx,ix)S(qx,jx) w(q) JxW(q)
// is symmetric positive definite and depends only on the two unordered 1D
// index pairs {iz,jz} and {ix,jx}: 225 sums at k = 4, each stored in one or two
// places of the packed lower triangle, by sum factorisation over the pairs with
// the products S(q,a)S(q,b) tabulated once per block.  It is then inverted in
// place by the symmetric sweep operator (Gauss-Jordan restricted to the
// lower triangle; SPD, no pivoting), which leaves -M^{-1}.  The inverse is
// written out in full, transposed (it is symmetric).
//
// Bound by FP64 instructions, which cost a warp the same with one useful lane
// as with 32: with a warp per cell the pivots' divisions were a third of the
// kernel and 325 triangle entries left 8% of the lanes idle.  Four cells per
// warp share the division's instructions and fill the lanes (12,800 cells, k = 4:
// 0.47 -> 0.39 ms, the FP64 pipe 87% busy).  Fewer than 4096 cells leave SMs without
// warps; there a warp per cell is the shorter chain.

template <int K>
struct BlockInvCfg {
  static constexpr int NN = K + 1, NQ = 2 * K + 1, NN2 = NN * NN, NQ2 = NQ * NQ;
  static constexpr int NP = NN * (NN + 1) / 2;        // 1D pairs a <= b
  static constexpr int NTRI = NN2 * (NN2 + 1) / 2;    // packed lower triangle
  // per cell: the triangle, the quadrature weights, and the x-contracted
  // weights, whose space first holds the x-contracted weight field; the pivot
  // columns reuse the space of the last two.  8 mod 16 values: two groups'
  // equal offsets fall into different halves of the banks
  static constexpr int TBX = NQ * (NP > NN ? NP : NN);
  static constexpr int PER = (NTRI + NQ2 + TBX + 7) / 16 * 16 + 8;
  // block tables: S products [NQ][NP], then byte tables of triangle indices
  static constexpr int TAB_BYTES = ((NQ * NP) * 8 + 2 * NTRI + 7) / 8 * 8;
  template <typename T>
  static size_t smem(int cells) { return TAB_BYTES + sizeof(T) * (size_t)cells * PER; }
};

__device__ __forceinline__ int tri_index(int i, int j) {  // i >= j
  return i * (i + 1) / 2 + j;
}
__device__ __forceinline__ int sym_index(int i, int j) {
  return i >= j ? tri_index(i, j) : tri_index(j, i);
}

template <int K, typename T, int G, int BI_WARPS>
__global__ void __launch_bounds__(32 * BI_WARPS)
    k_block_inverse(T *__restrict__ out, const T *__restrict__ weight, MeshT<T> mesh) {
  using B = BlockInvCfg<K>;
  constexpr int NN = B::NN, NQ = B::NQ, NN2 = B::NN2, NQ2 = B::NQ2, NP = B::NP;
  constexpr int NTRI = B::NTRI, CPW = 32 / G;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T *ss = reinterpret_cast<T *>(sm_raw);                              // [NQ][NP]
  unsigned char *ti = sm_raw + (size_t)NQ * NP * sizeof(T);           // [NTRI] row
  unsigned char *tj = ti + NTRI;                                      // [NTRI] column
  T *wsm = reinterpret_cast<T *>(sm_raw + B::TAB_BYTES);
  // block tables
  for (int e = threadIdx.x; e < NQ * NP; e += blockDim.x) {
    const int q = e / NP, p = e - q * NP;
    int b = 0;
    while ((b + 1) * (b + 2) / 2 <= p) ++b;
    const int a = p - b * (b + 1) / 2;
    ss[e] = bS<K, T>(q, a) * bS<K, T>(q, b);
  }
  for (int e = threadIdx.x; e < NTRI; e += blockDim.x) {
    int i = 0;
    while ((i + 1) * (i + 2) / 2 <= e) ++i;
    ti[e] = (unsigned char)i;
    tj[e] = (unsigned char)(e - i * (i + 1) / 2);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, wl = threadIdx.x & 31, grp = wl / G, lane = wl & (G - 1);
  const int cw = (blockIdx.x * BI_WARPS + warp) * CPW;  // first cell of the warp
  if (cw >= mesh.nc) return;  // warp-uniform; only warp-level barriers below
  const int c = min(cw + grp, mesh.nc - 1);  // a spare group repeats the last cell
  T *M = wsm + (warp * CPW + grp) * B::PER;  // [NTRI] packed lower triangle
  T *wq = M + NTRI;              // [NQ2] w JxW at the quadrature points
  T *Tb = wq + NQ2;              // [NQ][NP] x-contracted weights
  T *tx = Tb;                    // [NN][NQ] x-contracted weight field, before Tb
  T *colk = wq, *cd = colk + NN2;  // [NN2] pivot column, and it over the pivot
  static_assert(2 * NN2 <= NQ2 + NQ * NP, "pivot columns fit the assembly's space");
  const T *J = mesh.jw + c * mesh.jw_stride;
  if (weight) {
    const T *wt = weight + (long)c * NN2;
    for (int e = lane; e < NN * NQ; e += G) {
      const int iz = e / NQ, qx = e - iz * NQ;
      T s = T(0.0);
#pragma unroll
      for (int ix = 0; ix < NN; ++ix) s = fma(bS<K, T>(qx, ix), wt[iz * NN + ix], s);
      tx[e] = s;
    }
    __syncwarp();
    for (int q = lane; q < NQ2; q += G) {
      const int qz = q / NQ, qx = q - qz * NQ;
      T s = T(0.0);
#pragma unroll
      for (int iz = 0; iz < NN; ++iz) s = fma(bS<K, T>(qz, iz), tx[iz * NQ + qx], s);
      wq[q] = s * J[q];
    }
  } else {
    for (int q = lane; q < NQ2; q += G) wq[q] = J[q];
  }
  __syncwarp();
  for (int e = lane; e < NQ * NP; e += G) {
    const int qz = e / NP, p = e - qz * NP;
    T s = T(0.0);
#pragma unroll
    for (int qx = 0; qx < NQ; ++qx) s = fma(ss[qx * NP + p], wq[qz * NQ + qx], s);
    Tb[e] = s;
  }
  __syncwarp();
  for (int e = lane; e < NP * NP; e += G) {
    const int pz = e / NP, px = e - pz * NP;
    T s = T(0.0);
#pragma unroll
    for (int qz = 0; qz < NQ; ++qz) s = fma(ss[qz * NP + pz], Tb[qz * NP + px], s);
    const int zb = ti[pz], za = tj[pz], xb = ti[px], xa = tj[px];  // a <= b
    M[tri_index(zb * NN + xb, za * NN + xa)] = s;
    if (zb != za) M[tri_index(zb * NN + xa, za * NN + xb)] = s;
  }
  __syncwarp();
  // symmetric sweep on pivots k = 0..NN2-1:
  //   a_ij -= a_ik a_kj / a_kk (i, j != k);  a_ik = a_ik / a_kk;  a_kk = -1 / a_kk
  for (int k = 0; k < NN2; ++k) {
    const T d = T(1.0) / M[tri_index(k, k)];
    for (int i = lane; i < NN2; i += G) {
      const T a = M[sym_index(i, k)];
      colk[i] = a;
      cd[i] = a * d;
    }
    __syncwarp();
#pragma unroll 4
    for (int e = lane; e < NTRI; e += G) {
      const int i = ti[e], j = tj[e];
      if (i != k && j != k) M[e] = fma(-cd[i], colk[j], M[e]);
    }
    __syncwarp();
    for (int i = lane; i < NN2; i += G) M[sym_index(i, k)] = i == k ? -d : cd[i];
    __syncwarp();
  }
  for (int g = 0; g < CPW && cw + g < mesh.nc; ++g) {
    T *o = out + (long)(cw + g) * ainv_stride<K, T>(mesh.exact);
    const T *Mg = wsm + (warp * CPW + g) * B::PER;
    if constexpr (sizeof(T) == 4) {  // lower triangle, by rows or by tiles (ainv_stride)
      for (int e = wl; e < NTRI; e += 32)
        o[mesh.exact ? atile_index<K>(ti[e], tj[e]) : e] = -Mg[e];
    } else {
      for (int e = wl; e < NN2 * NN2; e += 32) {
        const int j = e / NN2, i = e - j * NN2;
        o[e] = -Mg[sym_index(i, j)];
      }
    }
  }
}

// dst[c][comp][i] = scale * sum_j Binv[c][i][j] src[c][comp][j]  (transposed storage)
template <int K, typename T>
__global__ void k_block_apply(T *__restrict__ dst, const T *__restrict__ src,
                              const T *__restrict__ binvT, int ncomp, T scale,
                              int nc) {
  constexpr int NN2 = (K + 1) * (K + 1);
  static_assert(sizeof(T) == 8, "full A^{-1} blocks are FP64 (FP32 stores a triangle)");
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (long)nc * NN2) return;
  const int c = (int)(g / NN2), i = (int)(g - (long)c * NN2);
  const T *B = binvT + (long)c * ainv_stride<K, T>();
  for (int comp = 0; comp < ncomp; ++comp) {
    const T *s = src + ((long)c * ncomp + comp) * NN2;
    T acc = T(0.0);
#pragma unroll 4
    for (int j = 0; j < NN2; ++j) acc = fma(B[j * NN2 + i], s[j], acc);
    dst[((long)c * ncomp + comp) * NN2 + i] = scale * acc;
  }
}

namespace {
template <int K, typename T>
int mass_launch(const OpView<T> &v, T *dst, const T *src, int ncomp, const T *weight,
                T scale) {
  using C = Cfg<K>;
  const int grid = (v.nc + C::CPB - 1) / C::CPB;
  const size_t sm = sizeof(T) * C::CPB * (3 * C::NN2 + 2 * C::NN * C::NQ);
  if (ncomp == 1 && !weight) k_mass<K, 1, false, T><<<grid, C::THREADS, sm, v.st>>>(dst, src, weight, scale, v.mesh);
  else if (ncomp == 1) k_mass<K, 1, true, T><<<grid, C::THREADS, sm, v.st>>>(dst, src, weight, scale, v.mesh);
  else if (!weight) k_mass<K, 2, false, T><<<grid, C::THREADS, sm, v.st>>>(dst, src, weight, scale, v.mesh);
  else k_mass<K, 2, true, T><<<grid, C::THREADS, sm, v.st>>>(dst, src, weight, scale, v.mesh);
  ATM_CHECK_LAUNCH("k_mass");
  return ATM_OK;
}

template <int K, typename T>
int invdiag_launch(const OpView<T> &v, T *out, int ncomp, const T *weight, T scale) {
  using C = Cfg<K>;
  const int grid = (v.nc + C::CPB - 1) / C::CPB;
  const size_t sm = sizeof(T) * C::CPB * (C::NN2 + C::NN * C::NQ);
  if (weight) k_invdiag<K, true, T><<<grid, C::THREADS, sm, v.st>>>(out, ncomp, weight, scale, v.mesh);
  else k_invdiag<K, false, T><<<grid, C::THREADS, sm, v.st>>>(out, ncomp, weight, scale, v.mesh);
  ATM_CHECK_LAUNCH("k_invdiag");
  return ATM_OK;
}

template <int K, typename T>
int block_inverse_launch(const OpView<T> &v, T *out, const T *weight) {
  // a warp per cell, or several.  At k = 5 four cells per warp take 33 KB of shared
  // memory, so that an SM holds one block of four warps: slower than a warp per
  // cell.  Two cells keep twelve warps: 2254 us at 28800 cells, a warp per cell
  // 2476.  Their lines cross between 4700 cells (564 / 447 us) and 7200 (589 / 694)
  const bool one = v.nc < (K == 5 ? 6000 : 4096);
  constexpr int G = K == 5 ? 16 : 8, W = 4;
  const int warps = one ? 2 : W, cells = one ? 2 : W * (32 / G);
  const size_t sm = BlockInvCfg<K>::template smem<T>(cells);
  void (*fn)(T *, const T *, MeshT<T>) =
      one ? k_block_inverse<K, T, 32, 2> : k_block_inverse<K, T, G, W>;
  ATM_CUDA(allow_smem(fn, sm));
  fn<<<(v.nc + cells - 1) / cells, 32 * warps, sm, v.st>>>(out, weight, v.mesh);
  ATM_CHECK_LAUNCH("k_block_inverse");
  return ATM_OK;
}

template <int K, typename T>
int block_apply_launch(const OpView<T> &v, T *dst, const T *src, const T *binv, int ncomp,
                       T scale) {
  constexpr int NN2 = (K + 1) * (K + 1);
  const long n = (long)v.nc * NN2;
  const int threads = 256;
  const int grid = (int)((n + threads - 1) / threads);
  k_block_apply<K, T><<<grid, threads, 0, v.st>>>(dst, src, binv, ncomp, scale, v.nc);
  ATM_CHECK_LAUNCH("k_block_apply");
  return ATM_OK;
}
}  // namespace
int launch_B(const atm_ctx &c, double *dst, const double *p, double cB, int mode, double cC) {
  const double ns = (double)c.nc * c.nn2;
  // p read; B p written (2 comps); mode 1 reads dst too; mode 2 reads A^{-1}
  const double bytes = 8.0 * ns * (1 + 2 + (mode == 1 ? 2 : 0)) +
                       (mode == 2 ? 8.0 * c.nc * c.nn2 * c.nn2 : 0.0);
  const double flops = c.nc * fl_B(c.k, c.mesh.exact, mode == 2);
  TimedRegion tr(c, KF_B, bytes, flops);
  if (c.mesh.exact) return exact_B(schur_view(c), dst, p, cB, cC, mode);
  if (c.mesh.nhang > 0) return launch_B_hang(c, dst, p, cB, mode);
  ATM_DISPATCH_K(c.k, (B_launch<K, double, false>(schur_view(c), dst, p, cB, mode)));
}
int launch_CD(const atm_ctx &c, double *dst, const double *w, const double *p, double coeff,
              int mode, bool workspace) {
  const double ns = (double)c.nc * c.nn2;
  const bool wd = (mode == 1 || mode == 2);
  // w (2 comps) + pfix read, [p], [inverse diagonal], [dst read], dst written
  const double bytes = 8.0 * ns * (3 + (wd ? 1 : 0) + (mode == 2 ? 1 : 0) + (mode == 3 ? 1 : 0) + 1);
  const double flops = c.nc * fl_CD(c.k, c.mesh.exact, wd);
  TimedRegion tr(c, KF_CD, bytes, flops);
  if (c.mesh.exact) return exact_CD(schur_view(c, workspace), dst, w, p, coeff, mode, nullptr);
  if (c.mesh.nhang > 0) return launch_CD_hang(c, dst, w, p, coeff, mode);
  ATM_DISPATCH_K(c.k, (CD_launch<K, double, false>(schur_view(c), dst, w, p, coeff, mode)));
}
int launch_pfix_prep(const atm_ctx &c, const double *p) {
  // p read and copied; its products with the cofactors at the points of C (general
  // kernels: its values at the quadrature points) and its face traces written
  const double nc = (3 * c.k + 3) / 2, nn = c.nn;
  const double bytes =
      8.0 * c.nc * (2.0 * c.nn2 + (c.mesh.exact ? 4.0 * nc * nc : c.nq2) + 4.0 * c.nq);
  const double volume = c.mesh.exact ? 2.0 * (nn * nn * nc + nn * nc * nc) + 4.0 * nc * nc : fl_eval(c.k);
  TimedRegion tr(c, KF_PFIX_PREP, bytes, c.nc * (volume + 4.0 * fl_face(c.k)));
  if (c.mesh.exact) return exact_pfix(schur_view(c), p);
  if (int rc = vec_copy(c.stream, c.pres_fix, p, c.n_scalar())) return rc;
  ATM_DISPATCH_K(c.k, (pfix_prep_launch<K, double>(schur_view(c))));
}
int launch_mass(const atm_ctx &c, double *dst, const double *src, int ncomp,
                const double *weight, double scale) {
  const double ns = (double)c.nc * c.nn2;
  const double bytes = 8.0 * ns * (2 * ncomp + (weight ? 1 : 0));
  const double flops = c.nc * ((ncomp + (weight ? 1 : 0)) * fl_eval(c.k) +
                               ncomp * fl_integrate(c.k, false));
  TimedRegion tr(c, KF_MASS, bytes, flops);
  ATM_DISPATCH_K(c.k, (mass_launch<K, double>(schur_view(c), dst, src, ncomp, weight, scale)));
}
int launch_inv_diag(const atm_ctx &c, double *out, int ncomp, const double *weight,
                    double scale) {
  TimedRegion tr(c, KF_DIAG, 8.0 * c.nc * c.nn2 * (ncomp + (weight ? 1 : 0)), 0.0);
  ATM_DISPATCH_K(c.k, (invdiag_launch<K, double>(schur_view(c), out, ncomp, weight, scale)));
}
int launch_block_inverse(const atm_ctx &c, double *out, const double *weight) {
  const double nn = c.nn, nq = c.nq, nn2 = c.nn2;
  // weight read, inverse written; flops: mass assembly + Gauss-Jordan
  const double bytes = 8.0 * c.nc * (nn2 * (weight ? 1 : 0) + nn2 * nn2);
  const double flops = c.nc * (2.0 * (nq * nn * nn * nq + nn2 * nn2 * nq) + 2.0 * nn2 * nn2 * nn2);
  TimedRegion tr(c, KF_BLOCK_INV, bytes, flops);
  ATM_DISPATCH_K(c.k, (block_inverse_launch<K, double>(schur_view(c), out, weight)));
}
int launch_block_apply(const atm_ctx &c, double *dst, const double *src, const double *binv,
                       int ncomp, double scale) {
  const double nn2 = c.nn2;
  const double bytes = 8.0 * c.nc * (nn2 * nn2 + 2.0 * ncomp * nn2);
  const double flops = 2.0 * c.nc * ncomp * nn2 * nn2;
  TimedRegion tr(c, KF_BLOCK_APPLY, bytes, flops);
  ATM_DISPATCH_K(c.k, (block_apply_launch<K, double>(schur_view(c), dst, src, binv, ncomp, scale)));
}

// ---- launchers on a multigrid level (untimed; float or double) -----------
template <typename T>
int level_B(const LevelViewT<T> &v, T *dst, const T *p, T cB, T cC) {
  if (v.mesh.exact) return exact_B(v, dst, p, cB, cC, 2);
  if (v.mesh.nhang > 0) return level_B_hang<T>(v, dst, p, cB, 2);
  if constexpr (sizeof(T) == 4) return general_B_f(v, dst, p, cB);
  else ATM_DISPATCH_K(v.k, (B_launch<K, T, false>(v, dst, p, cB, 2)));
}
template <typename T>
int level_CD(const LevelViewT<T> &v, T *dst, const T *w, const T *p, T cC, int mode) {
  if (v.mesh.exact) return exact_CD(v, dst, w, p, cC, mode, nullptr);
  if (v.mesh.nhang > 0) return level_CD_hang<T>(v, dst, w, p, cC, mode, nullptr);
  if constexpr (sizeof(T) == 4) return general_CD_f(v, dst, w, p, cC, mode, nullptr);
  else ATM_DISPATCH_K(v.k, (CD_launch<K, T, false>(v, dst, w, p, cC, mode)));
}
template <typename T>
int level_CD_cheb(const LevelViewT<T> &v, const T *w, T cC, const ChebArgs<T> &ch) {
  if (v.mesh.exact) return exact_CD(v, (T *)nullptr, w, ch.x, cC, 4, &ch);
  if (v.mesh.nhang > 0) return level_CD_hang<T>(v, nullptr, w, ch.x, cC, 4, &ch);
  if constexpr (sizeof(T) == 4) return general_CD_f(v, nullptr, w, ch.x, cC, 4, &ch);
  else ATM_DISPATCH_K(v.k, (CD_launch<K, T, false>(v, nullptr, w, ch.x, cC, 4, &ch)));
}
template <typename T>
int level_pfix_prep(const LevelViewT<T> &v) {
  if (v.mesh.exact) return exact_pfix(v, v.pfix);
  ATM_DISPATCH_K(v.k, (pfix_prep_launch<K, T>(v)));
}
template <typename T>
int level_inv_diag(const LevelViewT<T> &v, T *out, T scale) {
  ATM_DISPATCH_K(v.k, (invdiag_launch<K, T>(v, out, 1, (const T *)nullptr, scale)));
}
template <typename T>
int level_block_inverse(const LevelViewT<T> &v, T *out, const T *weight) {
  ATM_DISPATCH_K(v.k, (block_inverse_launch<K, T>(v, out, weight)));
}
#define ATM_LEVEL_INST(T)                                                                   \
  template int level_B<T>(const LevelViewT<T> &, T *, const T *, T, T);                     \
  template int level_CD<T>(const LevelViewT<T> &, T *, const T *, const T *, T, int);       \
  template int level_pfix_prep<T>(const LevelViewT<T> &);                                   \
  template int level_CD_cheb<T>(const LevelViewT<T> &, const T *, T, const ChebArgs<T> &);   \
  template int level_inv_diag<T>(const LevelViewT<T> &, T *, T);                            \
  template int level_block_inverse<T>(const LevelViewT<T> &, T *, const T *);
ATM_LEVEL_INST(float)
ATM_LEVEL_INST(double)

}  // namespace atm