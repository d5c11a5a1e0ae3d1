// FP64 instantiations of the Schur kernels for mappings of degree <= 2 on
// conforming meshes, and what all of them share: the 1D tables and the
// geometry tables (schur_exact.cuh explains the point sets).
#include "schur_exact.cuh"

namespace atm {

int upload_exact_f(const double *t);
int upload_contract_rhs(const double *t);
int upload_contract_hang_rhs(const double *t);
int upload_exact_hang(const double *t);
int upload_exact_hang_f(const double *t);

namespace {
// Gauss points and weights of the three point sets, passed by value
struct ExactPts {
  double x[EO_SETS][NQ_MAX], w[EO_SETS][NQ_MAX];
};

ExactPts exact_points(int k) {
  ExactPts P{};
  const int np[EO_SETS] = {k + 1, (3 * k + 3) / 2, 2 * k + 1};
  for (int s = 0; s < EO_SETS; ++s) {
    std::vector<double> x, w;
    gauss_nodes(np[s], x, w);
    for (int q = 0; q < np[s]; ++q) {
      P.x[s][q] = x[q];
      P.w[s][q] = w[q];
    }
  }
  return P;
}

// factor of the averages in the face terms of C
constexpr double C_FACE = 0.5 * GAS_GAMMA / (GAS_GAMMA - 1.0);

// degree-2 Lagrange basis on {0, 1/2, 1}
__device__ __forceinline__ void lag2(double x, double (&v)[3], double (&d)[3]) {
  v[0] = (2.0 * x - 1.0) * (x - 1.0);
  v[1] = 4.0 * x * (1.0 - x);
  v[2] = x * (2.0 * x - 1.0);
  d[0] = 4.0 * x - 3.0;
  d[1] = 4.0 - 8.0 * x;
  d[2] = 4.0 * x - 1.0;
}
// Jacobian [x_xi, x_eta, z_xi, z_eta] of the degree-2 mapping X[3][3][2],
// from the offsets to its centre node (coordinates are large, cells small)
__device__ __forceinline__ void jac2(const double *__restrict__ X, double xi, double eta,
                                     double (&J)[4]) {
  double vx[3], dx[3], ve[3], de[3];
  lag2(xi, vx, dx);
  lag2(eta, ve, de);
  J[0] = J[1] = J[2] = J[3] = 0.0;
  const double cx = X[8], cz = X[9];
  for (int e = 0; e < 3; ++e)
    for (int a = 0; a < 3; ++a) {
      const double x = X[(e * 3 + a) * 2] - cx, z = X[(e * 3 + a) * 2 + 1] - cz;
      J[0] += x * (dx[a] * ve[e]);
      J[1] += x * (vx[a] * de[e]);
      J[2] += z * (dx[a] * ve[e]);
      J[3] += z * (vx[a] * de[e]);
    }
}
// outward normal times the face weight of face f at parameter t
__device__ __forceinline__ void face2(const double *__restrict__ X, int f, double t, double w,
                                      double &n0, double &n1) {
  double J[4];
  jac2(X, f == 0 ? 0.0 : f == 1 ? 1.0 : t, f == 2 ? 0.0 : f == 3 ? 1.0 : t, J);
  const double s = (f & 1) ? w : -w;
  n0 = s * (f < 2 ? J[3] : -J[2]);
  n1 = s * (f < 2 ? -J[1] : J[0]);
}

// one thread per (cell, table entry)
template <typename T>
__global__ void k_exact_tables(MeshT<T> m, const double *__restrict__ map2, ExactPts P, int k,
                               bool own_jw) {
  const int nn = k + 1, nc = (3 * k + 3) / 2, nq = 2 * k + 1;
  const int n1 = nn * nn, n2 = n1 + nc * nc, n3 = n2 + 4 * nn, n4 = n3 + 4 * nq;
  const int n5 = n4 + (own_jw ? nq * nq : 0);
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (long)m.nc * n5) return;
  const long c = g / n5;
  int e = (int)(g - c * n5);
  const double *X = map2 + c * 18;
  double J[4];
  if (e >= n4) {  // det J x weight at the (2k+1)^2 points, index qz * nq + qx
    e -= n4;
    const int qz = e / nq, qx = e - qz * nq;
    jac2(X, P.x[2][qx], P.x[2][qz], J);
    m.jw[c * nq * nq + e] = (T)((J[0] * J[3] - J[1] * J[2]) * (P.w[2][qx] * P.w[2][qz]));
  } else if (e < n2) {  // volume points, index qx * np + qz
    const int s = e < n1 ? 0 : 1, np = s ? nc : nn;
    if (s) e -= n1;
    const int qx = e / np, qz = e - qx * np;
    jac2(X, P.x[s][qx], P.x[s][qz], J);
    const double w = P.w[s][qx] * P.w[s][qz];
    // cofactors times the weight: (xi, eta) tested with d/dx, then with d/dz
    const double cof[4] = {J[3] * w, -J[2] * w, -J[1] * w, J[0] * w};
    const long o = (c * np * np + e) * 4;
    for (int d = 0; d < 4; ++d) {
      if (s) m.gC[o + d] = (T)(GAS_GAMMA / (GAS_GAMMA - 1.0) * cof[d]);
      else m.gB[o + d] = (T)cof[d];
    }
    if (s) m.gJ[c * np * np + e] = (T)((J[0] * J[3] - J[1] * J[2]) * w / (GAS_GAMMA - 1.0));
  } else {
    const bool B = e < n3;
    const int np = B ? nn : nq, s = B ? 0 : 2;
    e -= B ? n2 : n3;
    const int f = e / np, q = e - f * np;
    double a, b;
    face2(X, f, P.x[s][q], P.w[s][q], a, b);
    T *o = (B ? m.fB : m.fC) + ((c * 4 + f) * np + q) * 2;
    const double h = B ? 0.5 : C_FACE;
    o[0] = (T)(h * a);
    o[1] = (T)(h * b);
  }
}
// subfaces of the coarse side of hanging faces: hcf[h] = 4 cell + face
template <typename T>
__global__ void k_exact_hang_tables(MeshT<T> m, const double *__restrict__ map2,
                                    const int *__restrict__ hcf, ExactPts P, int k) {
  const int nn = k + 1, nq = 2 * k + 1, per = nn + nq;
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (long)m.nhang * 2 * per) return;
  const long hs = g / per;
  int q = (int)(g - hs * per);
  const bool B = q < nn;
  if (!B) q -= nn;
  const int cf = hcf[hs >> 1], sub = (int)(hs & 1), s = B ? 0 : 2;
  double a, b;
  face2(map2 + (long)(cf >> 2) * 18, cf & 3, 0.5 * (P.x[s][q] + sub), 0.5 * P.w[s][q], a, b);
  T *o = (B ? m.hB + hs * nn * 2 : m.hC + hs * nq * 2) + q * 2;
  const double h = B ? 0.5 : C_FACE;
  o[0] = (T)(h * a);
  o[1] = (T)(h * b);
}
}  // namespace

// 1D tables of every degree to the constant banks of the translation units that
// contract with them
int upload_exact_all() {
  std::vector<double> t(EO_DOUBLES + SUB_DOUBLES, 0.0);
  for (int k = 1; k <= KMAX; ++k) {
    const std::vector<double> gll = gll_nodes(k);
    const int np[EO_SETS] = {k + 1, (3 * k + 3) / 2, 2 * k + 1};
    std::vector<double> x, w, S(k + 1), D(k + 1);
    for (int s = 0; s < EO_SETS; ++s) {
      gauss_nodes(np[s], x, w);
      for (int q = 0; q < (np[s] + 1) / 2; ++q) {
        lagrange_eval(gll, x[q], S.data(), D.data());
        for (int i = 0; i <= k / 2; ++i) {
          const double m[4] = {0.5 * (S[i] + S[k - i]), 0.5 * (S[i] - S[k - i]),
                               0.5 * (D[i] + D[k - i]), 0.5 * (D[i] - D[k - i])};
          for (int v = 0; v < 4; ++v)
            t[(((k * EO_SETS + s) * 4 + v) * EO_Q + q) * EO_I + i] = m[v];
        }
      }
      if (s == 1) continue;
      for (int h = 0; h < 2; ++h)
        for (int q = 0; q < np[s]; ++q) {
          lagrange_eval(gll, 0.5 * (x[q] + h), S.data(), nullptr);
          for (int i = 0; i <= k; ++i)
            t[EO_DOUBLES + (((k * 2 + (s ? 1 : 0)) * 2 + h) * NQ_MAX + q) * NN_MAX + i] = S[i];
        }
    }
  }
  return upload_exact_here(t.data()) || upload_exact_f(t.data()) || upload_exact_hang(t.data()) ||
         upload_exact_hang_f(t.data()) || upload_contract_rhs(t.data()) ||
         upload_contract_hang_rhs(t.data());
}

template <typename T>
void exact_mesh_free(MeshT<T> &m) {
  if (!m.qgeo) cudaFree(m.jw);
  m.jw = nullptr;
  T **v[] = {&m.gB, &m.fB, &m.gC, &m.gJ, &m.fC, &m.hB, &m.hC};
  for (T **p : v) {
    cudaFree(*p);
    *p = nullptr;
  }
  m.exact = false;
}

// geometry tables of the mapping at degree 2 (map2 as MeshT::map2, host)
template <typename T>
int exact_mesh_build(MeshT<T> &m, const double *map2, const std::vector<int> &hcf,
                     cudaStream_t st) {
  const int k = m.k, nn = k + 1, nc = (3 * k + 3) / 2, nq = 2 * k + 1;
  const size_t n = m.nc;
  T **ptr[] = {&m.gB, &m.fB, &m.gC, &m.gJ, &m.fC, &m.hB, &m.hC};
  const size_t len[] = {n * nn * nn * 4, n * 8 * nn, n * nc * nc * 4, n * nc * nc, n * 8 * nq,
                        (size_t)m.nhang * 4 * nn, (size_t)m.nhang * 4 * nq};
  for (int i = 0; i < 7; ++i)
    if (len[i]) ATM_CUDA(cudaMalloc(ptr[i], len[i] * sizeof(T)));
  const bool own_jw = !m.qgeo;  // a level without the full geometry table
  if (own_jw) {
    ATM_CUDA(cudaMalloc(&m.jw, n * nq * nq * sizeof(T)));
    m.jw_stride = nq * nq;
  }
  const ExactPts P = exact_points(k);
  double *dm = nullptr;
  int *dh = nullptr;
  ATM_CUDA(cudaMalloc(&dm, n * 18 * sizeof(double)));
  cudaError_t e = cudaMemcpyAsync(dm, map2, n * 18 * sizeof(double), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    const long items =
        (long)n * (nn * nn + nc * nc + 4 * nn + 4 * nq + (own_jw ? nq * nq : 0));
    k_exact_tables<T><<<(unsigned)((items + 255) / 256), 256, 0, st>>>(m, dm, P, k, own_jw);
    g_kernel_launches.fetch_add(1);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && m.nhang > 0) {
    e = cudaMalloc(&dh, hcf.size() * sizeof(int));
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(dh, hcf.data(), hcf.size() * sizeof(int), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
      const long items = (long)m.nhang * 2 * (nn + nq);
      k_exact_hang_tables<T><<<(unsigned)((items + 255) / 256), 256, 0, st>>>(m, dm, dh, P, k);
      g_kernel_launches.fetch_add(1);
      e = cudaGetLastError();
    }
  }
  const cudaError_t s = cudaStreamSynchronize(st);  // pageable sources, temporary buffers
  cudaFree(dm);
  cudaFree(dh);
  if (e == cudaSuccess) e = s;
  if (e != cudaSuccess) return cuda_fail(e, "geometry tables of the Schur kernels");
  m.exact = true;
  return ATM_OK;
}
template void exact_mesh_free<double>(MeshT<double> &);
template void exact_mesh_free<float>(MeshT<float> &);
template int exact_mesh_build<double>(MeshT<double> &, const double *, const std::vector<int> &,
                                      cudaStream_t);
template int exact_mesh_build<float>(MeshT<float> &, const double *, const std::vector<int> &,
                                     cudaStream_t);

int exact_B_hang(const OpView<double> &o, double *dst, const double *p, double cB, double cC,
                 int mode);
int exact_CD_hang(const OpView<double> &o, double *dst, const double *w, const double *p,
                  double cC, int mode, const ChebArgs<double> *ch);

int exact_B(const OpView<double> &o, double *dst, const double *p, double cB, double cC,
            int mode) {
  if (o.mesh.nhang > 0) return exact_B_hang(o, dst, p, cB, cC, mode);
  ATM_DISPATCH_K(o.k, (exact_B_launch<K, double, false>(o, dst, p, cB, cC, mode)));
}
int exact_CD(const OpView<double> &o, double *dst, const double *w, const double *p, double cC,
             int mode, const ChebArgs<double> *ch) {
  if (o.mesh.nhang > 0) return exact_CD_hang(o, dst, w, p, cC, mode, ch);
  ATM_DISPATCH_K(o.k, (exact_CD_launch<K, double, false>(o, dst, w, p, cC, mode, ch)));
}
int exact_pfix(const OpView<double> &o, const double *src) {
  ATM_DISPATCH_K(o.k, (exact_pfix_launch<K, double>(o, src)));
}

}  // namespace atm
