// Explicit IMEX stage right-hand sides (FP64), templated on the polynomial
// degree K, the IMEX stage ST and the equation KIND:
//   0 rho      : euler_operator.h:344-473 (cell), 478-692 (face), no boundary
//   1 momentum : euler_operator.h:1622-1886 (cell), 1891-2184 (face),
//                2189-2305 (wall, p_D = p)
//   2 energy   : euler_operator.h:745-1007 (cell), 1012-1361 (face), no boundary
//
// 2D form of the reference's 3D operators: gravity acts along -e_z with the
// factor a^2/r^2 = 1 (euler_operator.h:790-811 on a Cartesian domain).
//
// Each right-hand side has face and cell kernels, bound by their FP64
// instructions:
//   * k_rhs_face integrates the numerical flux of every face once.  The fluxes
//     are conservative (the reference's "+" and "-" contributions are one
//     expression with the sides swapped and n -> -n), so of the two sides of a
//     conforming face only the odd local face (1: x = 1, 3: z = 1) is
//     integrated and its nodal integrals go to both cells, with opposite
//     signs.  Walls and hanging faces are integrated from each of their sides,
//     with that side's geometry.
//   * k_rhs_cell evaluates the fields row by row and column by column (one
//     thread per 1D contraction, contract.cuh), forms the cell integrals and
//     adds the face integrals.
//
// The integrals pass from one kernel to the other in dst itself (FaceWay): a
// right-hand side writes nothing but its destination, so that calls on one
// handle may overlap, on several streams, threads or branches of a graph.
// A face trace takes 35 FP64 instructions per field and stage state, a face
// point about 20: integrating a face from both cells would cost a quarter of
// the whole right-hand side.  Runs are bitwise reproducible.
// Measured on GB300, the three right-hand sides of the last stage at 51,200
// cells, k = 4: 5.82 -> 3.99 ms against one kernel per equation with every
// face integrated twice and the x-contractions done point by point (the cell
// kernels keep the FP64 pipe 83-85% busy); 3239 cells, k = 3, second stage:
// 232 -> 192 us.
//
// The reference integrates with 2k+1 points.  The momentum flux (degree 4k+1
// on a degree-2 mapping) needs them all, the energy flux more; the density
// flux rho u cof grad v has degree 3k+1 and takes floor((3k+3)/2) points where
// the mesh has the tables of that set (`exact`, mapping degree <= 2).
#pragma once
#include "contract.cuh"

namespace atm {

template <int KIND>
struct RhsKind {
  static constexpr int NF = KIND == 0 ? 3 : 4;     // fields of a stage state: rho, u, [p]
  static constexpr int PER = KIND == 0 ? 2 : 3;    // source vectors of a stage state
  static constexpr int NCOMP = KIND == 1 ? 2 : 1;  // output components
};

// =============================================================== faces ===
// Traces of a cell's field on a face: at all 2k+1 points of the face or of its
// subface `sub` (>= 0), or at one point of it whose basis row is given.
template <int K>
struct LineTrace {
  int f, sub;
  __device__ __forceinline__ void operator()(const double *cell, double (&v)[2 * K + 1]) const {
    own_or_sub<K>(cell, f, sub, v);
  }
};
template <int K>
struct PointTrace {
  int f;
  const double *row;
  __device__ __forceinline__ void operator()(const double *cell, double (&v)[1]) const {
    double t[K + 1], s = 0.0;
    trace<K>(cell, f, t);
#pragma unroll
    for (int i = 0; i <= K; ++i) s = fma(row[i], t[i], s);
    v[0] = s;
  }
};

// How the face integrals reach dst.
//   FACE_HELD: all faces are integrated first and the cell kernel reads its cells'
//     values before it overwrites them.  With k >= 3 a cell's (k+1)^2 values hold
//     its 4 (k+1) face integrals in slots of their own.  With k <= 2 they do not
//     fit: dst is zeroed and a node gets the sum of its face integrals, at most
//     two (in a corner), by atomics; 0 + a + b does not depend on their order.
//   FACE_ADD_X, FACE_ADD_Z: for a dst that is also a source, which must not be
//     written before the cell kernel has read it.  The cell kernel goes first,
//     then the x-faces and the z-faces add to the nodes they touch, in two
//     launches (the two meet in the corner nodes).  For k <= 2 this order took 310
//     instead of 250 us at 8192 cells, k = 2, third stage.
enum FaceWay { FACE_HELD = 0, FACE_ADD_X = 1, FACE_ADD_Z = 2 };
template <int K>
constexpr bool FACE_SLOTS = K >= 3;
template <int K>  // values per cell and component that hold face integrals
constexpr int FACE_VALUES = FACE_SLOTS<K> ? 4 * (K + 1) : (K + 1) * (K + 1);

// local faces that a launch takes of each parity and cell, and the n-th of them
__device__ __forceinline__ int way_faces(int way) { return way == FACE_HELD ? 2 : 1; }
__device__ __forceinline__ int way_face(int way, int n, int odd) {
  return (way == FACE_HELD ? 2 * n : way == FACE_ADD_X ? 0 : 2) + odd;
}

// nodal integral i of component `comp` over face f of cell c
template <int K, int NCOMP>
__device__ __forceinline__ void face_put(double *__restrict__ dst, int way, int c, int f, int comp,
                                         int i, double v) {
  constexpr int NN = K + 1, NN2 = NN * NN;
  double *b = dst + ((long)c * NCOMP + comp) * NN2;
  double *node = b + (f < 2 ? i * NN + f * K : (f - 2) * K * NN + i);
  if (way != FACE_HELD) *node += v;
  else if (FACE_SLOTS<K>) b[f * NN + i] = v;
  else atomicAdd(node, v);
}

// F[comp][q] += numerical flux of all stage states at NQ points of one face,
// outward of cell c, times the face weight.  n0, n1: normal times weight; to,
// tn: traces of this cell and of the neighbour.
template <int K, int ST, int KIND, int NQ, typename Trace>
__device__ __forceinline__ void face_flux(const SrcPtrs &src, const StageCoef &co, int c, int nb,
                                          const Trace &to, const Trace &tn,
                                          const double (&n0)[NQ], const double (&n1)[NQ],
                                          double (&F)[RhsKind<KIND>::NCOMP][NQ]) {
  constexpr int NN2 = (K + 1) * (K + 1), PER = RhsKind<KIND>::PER;
  constexpr double IG = 1.0 / (GAS_GAMMA - 1.0), HGF = GAS_GAMMA * IG;
  constexpr bool MIXED = KIND == 2 && ST == 2;  // stage 2 mixes the states' velocities
  double xo[MIXED ? NQ : 1], zo[MIXED ? NQ : 1], xn[MIXED ? NQ : 1], zn[MIXED ? NQ : 1];
#pragma unroll
  for (int j = 0; j < ST; ++j) {
    const double *sr = src.p[PER * j], *su = src.p[PER * j + 1];
    double r[NQ], ux[NQ], uz[NQ], p[NQ], un[NQ];
    to(sr + (long)c * NN2, r);
    to(su + (long)c * 2 * NN2, ux);
    to(su + ((long)c * 2 + 1) * NN2, uz);
    if (KIND > 0) to(src.p[PER * j + 2] + (long)c * NN2, p);
    double vr[NQ], vx[NQ], vz[NQ], vp[NQ];
    tn(sr + (long)nb * NN2, vr);
    tn(su + (long)nb * 2 * NN2, vx);
    tn(su + ((long)nb * 2 + 1) * NN2, vz);
    if (KIND > 0) tn(src.p[PER * j + 2] + (long)nb * NN2, vp);
#pragma unroll
    for (int q = 0; q < NQ; ++q) un[q] = fma(ux[q], n0[q], uz[q] * n1[q]);
    if constexpr (KIND == 0) {
      const double h = 0.5 * co.ca[j] * co.dt;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const double um = fma(vx[q], n0[q], vz[q] * n1[q]);
        const double t = fma(abs_max(un[q], um), r[q] - vr[q], fma(r[q], un[q], vr[q] * um));
        F[0][q] = fma(h, t, F[0][q]);
      }
    } else if constexpr (KIND == 1) {
      const double h = 0.5 * co.ca[j] * co.dt, hp = 0.5 * co.ct[j] * co.dt / (co.Ma * co.Ma);
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const double um = fma(vx[q], n0[q], vz[q] * n1[q]);
        const double lam = abs_max(un[q], um);
        const double a0 = r[q] * ux[q], a1 = r[q] * uz[q], b0 = vr[q] * vx[q], b1 = vr[q] * vz[q];
        const double t0 = fma(lam, a0 - b0, fma(a0, un[q], b0 * um));
        const double t1 = fma(lam, a1 - b1, fma(a1, un[q], b1 * um));
        const double ps = hp * (p[q] + vp[q]);
        F[0][q] = fma(h, t0, fma(ps, n0[q], F[0][q]));
        F[1][q] = fma(h, t1, fma(ps, n1[q], F[1][q]));
      }
    } else {
      // per side s = k1 rho |u|^2 + k2 p (the flux over u.n) and t = k1 rho
      // |u|^2 + k3 p (what jumps); stage 3 jumps the total rho E
      // (euler_operator.h:1290,1313,1336), where the enthalpy carries the
      // explicit weight; the division by rho in the reference's E cancels
      const double wa = co.ca[j] * co.dt, we = ST == 3 ? wa : co.ct[j] * co.dt;
      const double k1 = 0.25 * wa * co.Ma * co.Ma, k2 = 0.5 * HGF * we, k3 = 0.5 * IG * we;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const double um = fma(vx[q], n0[q], vz[q] * n1[q]);
        const double lam = abs_max(un[q], um);
        const double a = k1 * r[q], b = k1 * vr[q];
        const double ka = a * fma(ux[q], ux[q], uz[q] * uz[q]);
        const double kb = b * fma(vx[q], vx[q], vz[q] * vz[q]);
        double ja = ka, jb = kb;
        if constexpr (MIXED) {
          if (j == 0) {
            xo[q] = ux[q]; zo[q] = uz[q]; xn[q] = vx[q]; zn[q] = vz[q];
          } else {  // the reference's mixed kinetic jump (euler_operator.h:1182-1183)
            ja = a * fma(ux[q], xo[q], uz[q] * zo[q]);
            jb = b * fma(vx[q], xn[q], vz[q] * zn[q]);
          }
        }
        F[0][q] = fma(fma(k2, p[q], ka), un[q], F[0][q]);
        F[0][q] = fma(fma(k2, vp[q], kb), um, F[0][q]);
        F[0][q] = fma(lam, fma(k3, p[q], ja) - fma(k3, vp[q], jb), F[0][q]);
      }
    }
  }
}

// Nodal integrals of the outward flux; one thread per face, the odd local faces
// first, then the even ones that are not the other side of a conforming face
// (walls of the momentum equation, hanging faces).
template <int K, int ST, int KIND, bool HG>
__global__ void __launch_bounds__(64)
    k_rhs_face(double *__restrict__ dst, int way, SrcPtrs src, StageCoef co, Mesh mesh) {
  constexpr int NN = K + 1, NN2 = NN * NN, NQ = 2 * K + 1, NCOMP = RhsKind<KIND>::NCOMP;
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long half = (long)way_faces(way) * mesh.nc;
  const bool even = g >= half;
  const long e = even ? g - half : g;
  if (e >= half) return;
  const int c = (int)(way == FACE_HELD ? e >> 1 : e);
  const int f = way_face(way, (int)(e & 1), even ? 0 : 1);
  const int nb = mesh.nbr[c * 4 + f], nfc = mesh.nbrf[c * 4 + f], nf = nfc & 3;
  if (nb < 0 && KIND != 1) return;
  const int code = HG && nb >= 0 ? nfc >> 2 : 0;
  if (even && nb >= 0 && code == 0) return;  // the neighbour's odd face
  if (mesh.dts) co.dt *= mesh.dts[c];  // per-member time step
  double o[NCOMP][NN];
  double n0[NQ], n1[NQ], F[NCOMP][NQ];
  if (!HG || code < 3) {
    const double *fg = mesh.fgeo + ((long)c * 4 + f) * 3 * NQ;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      n0[q] = fg[q] * fg[2 * NQ + q];
      n1[q] = fg[NQ + q] * fg[2 * NQ + q];
#pragma unroll
      for (int d = 0; d < NCOMP; ++d) F[d][q] = 0.0;
    }
    if (KIND == 1 && nb < 0) {  // no-flux wall: only the pressure term with p_D = p
#pragma unroll
      for (int j = 0; j < ST; ++j) {
        double p[NQ];
        own_or_sub<K>(src.p[RhsKind<KIND>::PER * j + 2] + (long)c * NN2, f, -1, p);
        const double w = co.ct[j] * co.dt / (co.Ma * co.Ma);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          F[0][q] = fma(w * p[q], n0[q], F[0][q]);
          F[NCOMP - 1][q] = fma(w * p[q], n1[q], F[NCOMP - 1][q]);
        }
      }
    } else {
      face_flux<K, ST, KIND>(src, co, c, nb, LineTrace<K>{f, -1},
                             LineTrace<K>{nf, HG ? code - 1 : -1}, n0, n1, F);
    }
#pragma unroll
    for (int d = 0; d < NCOMP; ++d) eo_integ<K, 2, NQ, true, false>(F[d], F[d], o[d]);
  } else {
#pragma unroll
    for (int d = 0; d < NCOMP; ++d)
#pragma unroll
      for (int i = 0; i < NN; ++i) o[d][i] = 0.0;
    for (int h = 0; h < 2; ++h) {
      const double *fg = mesh.hgeo + ((long)nb * 2 + h) * 3 * NQ;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        n0[q] = fg[q] * fg[2 * NQ + q];
        n1[q] = fg[NQ + q] * fg[2 * NQ + q];
#pragma unroll
        for (int d = 0; d < NCOMP; ++d) F[d][q] = 0.0;
      }
      face_flux<K, ST, KIND>(src, co, c, mesh.hnb[nb * 2 + h], LineTrace<K>{f, h},
                             LineTrace<K>{nf, -1}, n0, n1, F);
#pragma unroll
      for (int d = 0; d < NCOMP; ++d) sub_integ_add<K, 1>(F[d], h, o[d]);
    }
  }
#pragma unroll
  for (int d = 0; d < NCOMP; ++d)
#pragma unroll
    for (int i = 0; i < NN; ++i) {
      face_put<K, NCOMP>(dst, way, c, f, d, i, -o[d][i]);
      if (nb >= 0 && code == 0) face_put<K, NCOMP>(dst, way, nb, nf, d, i, o[d][i]);
    }
}

// The same with one thread per face point, RHS_FPB faces per block: 5 instead of
// 4 FP64 instructions per trace value at k = 4, but nine times the threads.  A
// face per thread needs tens of thousands of faces to reach every quarter of
// every SM, each of which takes 64 clocks for an FP64 instruction whether one
// warp issues it or many.
constexpr int RHS_FPB = 16;
template <int K, int ST, int KIND, bool HG>
__global__ void __launch_bounds__(RHS_FPB *(2 * K + 1))
    k_rhs_face_points(double *__restrict__ dst, int way, SrcPtrs src, StageCoef co, Mesh mesh) {
  constexpr int NN = K + 1, NN2 = NN * NN, NQ = 2 * K + 1, NCOMP = RhsKind<KIND>::NCOMP;
  constexpr int NT = HG ? 3 : 1, NH = HG ? 2 : 1;
  // basis rows at the face's points, and at those of its two subfaces
  __shared__ double sS[NT][NQ][NN], sF[RHS_FPB][NH][NCOMP][NQ];
  for (int e = threadIdx.x; e < NQ * NN; e += blockDim.x) {  // S from its even-odd halves
    const int q = e / NN, i = e - q * NN, qq = q <= K ? q : NQ - 1 - q;
    const int ii = q <= K ? i : K - i, a = ii <= K / 2 ? ii : K - ii;
    const double E = CEo<double>::get(K, 2, 0, qq, a), O = CEo<double>::get(K, 2, 1, qq, a);
    sS[0][q][i] = ii <= K / 2 ? E + O : E - O;
    if (HG)
      for (int h = 0; h < 2; ++h) sS[HG ? 1 + h : 0][q][i] = CEo<double>::sub(K, 1, h, q, i);
  }
  __syncthreads();
  // odd conforming faces and walls; (momentum) even walls; hanging faces
  const int per = way_faces(way);
  const long nodd = (long)per * mesh.nc, neven = KIND == 1 ? nodd : 0;
  const long g0 = (long)blockIdx.x * RHS_FPB;
  const int lf = threadIdx.x / NQ, q = threadIdx.x - lf * NQ;
  auto face_of = [&](long id, int &c, int &f, int &code) {  // false: nothing to integrate
    const bool hang = id >= nodd + neven;
    if (hang) {
      id -= nodd + neven;
      if (!HG || id >= 2 * nodd) return false;
      c = (int)(per == 2 ? id >> 2 : id >> 1);
      f = way_face(way, (int)(id >> 1) & 1, (int)(id & 1));
    } else {
      const bool even = id >= nodd;
      const long e = even ? id - nodd : id;
      c = (int)(per == 2 ? e >> 1 : e);
      f = way_face(way, (int)(e & 1), even ? 0 : 1);
    }
    const int nb = mesh.nbr[c * 4 + f];
    code = HG && nb >= 0 ? mesh.nbrf[c * 4 + f] >> 2 : 0;
    if (hang) return code != 0;
    return nb < 0 ? KIND == 1 : (f & 1) && code == 0;
  };
  int c, f, code;
  if (face_of(g0 + lf, c, f, code)) {
    const int nb = mesh.nbr[c * 4 + f], nf = mesh.nbrf[c * 4 + f] & 3;
    if (mesh.dts) co.dt *= mesh.dts[c];  // per-member time step
    for (int h = 0; h < (HG && code == 3 ? 2 : 1); ++h) {
      const double *fg = (HG && code == 3 ? mesh.hgeo + ((long)nb * 2 + h) * 3 * NQ
                                          : mesh.fgeo + ((long)c * 4 + f) * 3 * NQ) + q;
      const double n0[1] = {fg[0] * fg[2 * NQ]}, n1[1] = {fg[NQ] * fg[2 * NQ]};
      double F[NCOMP][1];
#pragma unroll
      for (int d = 0; d < NCOMP; ++d) F[d][0] = 0.0;
      const PointTrace<K> to{f, sS[HG && code == 3 ? 1 + h : 0][q]};
      if (nb < 0) {  // no-flux wall: only the pressure term with p_D = p
#pragma unroll
        for (int j = 0; j < ST; ++j) {
          double p[1];
          to(src.p[RhsKind<KIND>::PER * j + 2] + (long)c * NN2, p);
          const double w = co.ct[j] * co.dt / (co.Ma * co.Ma) * p[0];
          F[0][0] = fma(w, n0[0], F[0][0]);
          F[NCOMP - 1][0] = fma(w, n1[0], F[NCOMP - 1][0]);
        }
      } else {
        const int cn = HG && code == 3 ? mesh.hnb[nb * 2 + h] : nb;
        face_flux<K, ST, KIND>(src, co, c, cn, to,
                               PointTrace<K>{nf, sS[HG && (code == 1 || code == 2) ? code : 0][q]},
                               n0, n1, F);
      }
#pragma unroll
      for (int d = 0; d < NCOMP; ++d) sF[lf][HG ? h : 0][d][q] = F[d][0];
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < RHS_FPB * NCOMP * NN; t += blockDim.x) {
    const int l = t / (NCOMP * NN), r = t - l * NCOMP * NN, d = r / NN, i = r - d * NN;
    if (!face_of(g0 + l, c, f, code)) continue;
    double o = 0.0;
    if (HG && code == 3) {
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int k = 0; k < NQ; ++k)
          o = fma(sS[HG ? 1 + h : 0][k][i], sF[l][HG ? h : 0][d][k], o);
    } else {
#pragma unroll
      for (int k = 0; k < NQ; ++k) o = fma(sS[0][k][i], sF[l][0][d][k], o);
    }
    face_put<K, NCOMP>(dst, way, c, f, d, i, -o);
    const int nb = mesh.nbr[c * 4 + f];
    if (nb >= 0 && code == 0)
      face_put<K, NCOMP>(dst, way, nb, mesh.nbrf[c * 4 + f] & 3, d, i, o);
  }
}

// =============================================================== cells ===
// x-interpolation of NF fields (rho; rho, u; or rho, u, p) of the block's
// cells: X[l][field][iz][NP], one row per thread
template <int K, int SET, int NP, int NF>
__device__ __forceinline__ void rhs_rows(double *__restrict__ X, int per, const double *r,
                                         const double *u, const double *p, int c0, int cnt) {
  constexpr int NN = K + 1;
  for (int e = threadIdx.x; e < cnt * NF * NN; e += blockDim.x) {
    const int l = e / (NF * NN), i = e - l * (NF * NN);
    const long c = c0 + l;
    const double *row = i < NN ? r + (c * NN + i) * NN
                        : i < 3 * NN ? u + (c * 2 * NN + (i - NN)) * NN
                                     : p + (c * NN + (i - 3 * NN)) * NN;
    double t[NN], v[NP];
#pragma unroll
    for (int a = 0; a < NN; ++a) t[a] = __ldg(row + a);
    eo_interp<K, SET>(t, v);
#pragma unroll
    for (int q = 0; q < NP; ++q) X[l * per + i * NP + q] = v[q];
  }
}
// z-interpolation of one field's column
template <int K, int SET, int NP>
__device__ __forceinline__ void rhs_col(const double *__restrict__ x, double (&v)[NP]) {
  double t[K + 1];
#pragma unroll
  for (int i = 0; i <= K; ++i) t[i] = x[i * NP];
  eo_interp<K, SET>(t, v);
}

// face integrals that output row iz adds; F: the cell's held values, [4][k+1]
// slots or node sums
template <int K>
__device__ __forceinline__ void rhs_face_rows(const double *__restrict__ F, int iz,
                                              double (&add)[K + 1]) {
  constexpr int NN = K + 1;
  if constexpr (FACE_SLOTS<K>) {
#pragma unroll
    for (int i = 0; i < NN; ++i) add[i] = 0.0;
    add[0] += F[iz];
    add[K] += F[NN + iz];
    if (iz == 0 || iz == K) {
      const double *Fz = iz == 0 ? F + 2 * NN : F + 3 * NN;
#pragma unroll
      for (int i = 0; i < NN; ++i) add[i] += Fz[i];
    }
  } else {
#pragma unroll
    for (int i = 0; i < NN; ++i) add[i] = F[iz * NN + i];
  }
}

// Threads (cell, column); `cpb` cells per block.  With `held`, dst holds the
// face integrals of its cells (FaceWay).
template <int K, int ST, int KIND, bool EX>
__global__ void __launch_bounds__(256)
    k_rhs_cell(double *dst, SrcPtrs src, StageCoef co, Mesh mesh, bool held, int cpb) {
  using E = Ex<K>;
  using R = RhsKind<KIND>;
  constexpr int NN = E::NN, NN2 = E::NN2, NCOMP = R::NCOMP, PER = R::PER;
  constexpr int SET = EX ? 1 : 2, NP = EX ? E::NC : E::NQ, XS = NN * NP, XC = R::NF * XS;
  constexpr double IG = 1.0 / (GAS_GAMMA - 1.0), HGF = GAS_GAMMA * IG;
  constexpr int FV = FACE_VALUES<K>;
  extern __shared__ double sm[];  // [cpb][NF][NN][NP], then (held) [cpb][NCOMP][FV]
  const int tid = threadIdx.x, l = tid / NP, col = tid - l * NP;
  const int c0 = blockIdx.x * cpb, cnt = min(cpb, mesh.nc - c0);
  const bool active = l < cnt;
  const long c = c0 + l;
  double *sF = sm + cpb * XC;
  if (held) {
    for (int e = tid; e < cnt * NCOMP * FV; e += blockDim.x) {
      const int lc = e / FV, i = e - lc * FV;
      // (density and energy have no boundary term: nothing is in a wall's slot)
      const bool wall = FACE_SLOTS<K> && KIND != 1 && mesh.nbr[(c0 + lc / NCOMP) * 4 + i / NN] < 0;
      sF[e] = wall ? 0.0 : dst[((long)c0 * NCOMP + lc) * NN2 + i];
    }
  }
  if (mesh.dts && active) co.dt *= mesh.dts[c];  // per-member time step
  const double M2 = co.Ma * co.Ma;
  double *x = sm + l * XC + col;
  // momentum: g00, g01 = g10, g11 and v0, v1; the others: gx, gz and v0
  double ga[NP], gb[NP], gc[KIND == 1 ? NP : 1], v0[NP], v1[KIND == 1 ? NP : 1];
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    ga[q] = gb[q] = v0[q] = 0.0;
    if (KIND == 1) gc[q] = v1[q] = 0.0;
  }
#pragma unroll
  for (int j = 0; j < ST; ++j) {
    rhs_rows<K, SET, NP, R::NF>(sm, XC, src.p[PER * j], src.p[PER * j + 1],
                                KIND > 0 ? src.p[PER * j + 2] : nullptr, c0, cnt);
    __syncthreads();
    if (active) {
      double r[NP], ux[NP], uz[NP], p[NP];
      rhs_col<K, SET>(x, r);
      rhs_col<K, SET>(x + XS, ux);
      rhs_col<K, SET>(x + 2 * XS, uz);
      if (KIND > 0) rhs_col<K, SET>(x + 3 * XS, p);
      const double wa = co.ca[j] * co.dt;
      if constexpr (KIND == 0) {
        // the tables of the smaller point set carry gamma/(gamma-1)
        const double w = EX ? wa / HGF : wa;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          if (j == 0) v0[q] = r[q];
          const double wr = w * r[q];
          ga[q] = fma(wr, ux[q], ga[q]);
          gb[q] = fma(wr, uz[q], gb[q]);
        }
      } else if constexpr (KIND == 1) {
        const double wp = co.ct[j] * co.dt / M2, wg = co.cg[j] * co.dt / (co.Fr * co.Fr);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          if (j == 0) {
            v0[q] = r[q] * ux[q];
            v1[q] = r[q] * uz[q];
          }
          v1[q] = fma(-wg, r[q], v1[q]);
          const double wr = wa * r[q], rx = wr * ux[q], rz = wr * uz[q];
          const double pp = wp * p[q];
          ga[q] += fma(rx, ux[q], pp);
          gb[q] = fma(rx, uz[q], gb[q]);
          gc[q] += fma(rz, uz[q], pp);
        }
      } else {
        // the reference forms E = p / ((gamma-1) rho) + Ma^2 |u|^2 / 2 and
        // uses rho E and rho (E - Ma^2 |u|^2 / 2) + p: the division cancels
        const double wgrav = co.cg[j] * co.dt * M2 / (co.Fr * co.Fr);
        const double wk = 0.5 * wa * M2, we = co.ct[j] * co.dt * HGF;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const double k = r[q] * fma(ux[q], ux[q], uz[q] * uz[q]);
          if (j == 0) v0[q] = fma(IG, p[q], 0.5 * M2 * k);  // rho E
          v0[q] = fma(-wgrav * r[q], uz[q], v0[q]);
          const double s = fma(wk, k, we * p[q]);
          ga[q] = fma(s, ux[q], ga[q]);
          gb[q] = fma(s, uz[q], gb[q]);
        }
      }
    }
    __syncthreads();
  }
  if constexpr (KIND == 1 && ST < 3) {  // implicit gravity of the density being solved for
    rhs_rows<K, SET, NP, 1>(sm, XC, src.p[PER * ST], nullptr, nullptr, c0, cnt);
    __syncthreads();
    if (active) {
      double r[NP];
      rhs_col<K, SET>(x, r);
      const double wg = co.cg[ST] * co.dt / (co.Fr * co.Fr);
#pragma unroll
      for (int q = 0; q < NP; ++q) v1[q] = fma(-wg, r[q], v1[q]);
    }
    __syncthreads();
  }
  if constexpr (KIND == 2) {
    if (src.p[PER * ST + 1]) {  // (not in a Picard loop's base) kinetic energy and gravity work of the fixed-point velocity
      rhs_rows<K, SET, NP, 3>(sm, XC, src.p[PER * ST], src.p[PER * ST + 1], nullptr, c0, cnt);
      __syncthreads();
      if (active) {
        double r[NP], ux[NP], uz[NP];
        rhs_col<K, SET>(x, r);
        rhs_col<K, SET>(x + XS, ux);
        rhs_col<K, SET>(x + 2 * XS, uz);
        const double wgrav = ST < 3 ? co.cg[ST < 3 ? ST : 0] * co.dt * M2 / (co.Fr * co.Fr) : 0.0;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          double t = 0.5 * M2 * fma(ux[q], ux[q], uz[q] * uz[q]);
          if (ST < 3) t = fma(wgrav, uz[q], t);
          v0[q] = fma(-t, r[q], v0[q]);
        }
      }
      __syncthreads();
    }
  }
  // fluxes to reference directions, z-integration; the results replace the
  // column's own values
  if (active) {
    double V[NP], Gx[NP], Ge[NP], a[NN], b[NN];
#pragma unroll
    for (int comp = 0; comp < NCOMP; ++comp) {
      if constexpr (EX) {
        const double *g = mesh.gC + (c * NP + col) * NP * 4, *jw = mesh.gJ + (c * NP + col) * NP;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const Vec4<double> w(g + 4 * q);
          V[q] = (GAS_GAMMA - 1.0) * v0[q] * __ldg(jw + q);  // gJ carries 1/(gamma-1)
          Gx[q] = fma(w.v[0], ga[q], w.v[2] * gb[q]);
          Ge[q] = fma(w.v[1], ga[q], w.v[3] * gb[q]);
        }
      } else {
        constexpr int NQ2 = NP * NP;
        const double *g = mesh.qgeo + c * 5 * NQ2 + col;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const double hx = comp == 0 ? ga[q] : gb[q];
          const double hz = KIND == 1 && comp == 1 ? gc[q] : gb[q];
          V[q] = (KIND == 1 && comp == 1 ? v1[q] : v0[q]) * __ldg(g + 4 * NQ2 + q * NP);
          Gx[q] = fma(__ldg(g + q * NP), hx, __ldg(g + NQ2 + q * NP) * hz);
          Ge[q] = fma(__ldg(g + 2 * NQ2 + q * NP), hx, __ldg(g + 3 * NQ2 + q * NP) * hz);
        }
      }
      eo_integ<K, SET, NP, true, true>(V, Ge, a);
      eo_integ<K, SET, NP, true, false>(Gx, Gx, b);
#pragma unroll
      for (int i = 0; i < NN; ++i) {
        x[2 * comp * XS + i * NP] = a[i];
        x[(2 * comp + 1) * XS + i * NP] = b[i];
      }
    }
  }
  __syncthreads();
  for (int e = tid; e < cnt * NCOMP * NN; e += blockDim.x) {
    const int lo = e / (NCOMP * NN), i = e - lo * (NCOMP * NN), comp = i / NN, iz = i - comp * NN;
    const double *y = sm + lo * XC + 2 * comp * XS + iz * NP;
    double a[NP], b[NP], out[NN], add[NN];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      a[q] = y[q];
      b[q] = y[XS + q];
    }
    eo_integ<K, SET, NP, true, true>(a, b, out);
    double *d = dst + ((long)(c0 + lo) * NCOMP + comp) * NN2 + iz * NN;
    if (held) {
      rhs_face_rows<K>(sF + (lo * NCOMP + comp) * FV, iz, add);
#pragma unroll
      for (int q = 0; q < NN; ++q) out[q] += add[q];
    }
#pragma unroll
    for (int q = 0; q < NN; ++q) d[q] = out[q];
  }
}

// dst = base - integrals of rho (Ma^2 |u|^2 / 2 + wgrav u_z) phi: what the
// energy right-hand side takes from the fixed-point velocity, the only part of
// it that changes from one Picard iteration to the next
// (Atmospheric_Flow.cc:1135-1153).  At 51,200 cells, k = 4 it takes a seventh
// of the time of the whole right-hand side.  Threads (cell, column).
template <int K>
__global__ void __launch_bounds__(256)
    k_rhs_kinetic(double *__restrict__ dst, const double *__restrict__ base,
                  const double *__restrict__ rho, const double *__restrict__ u, double wgrav,
                  double M2, Mesh mesh, int cpb) {
  constexpr int NN = K + 1, NP = 2 * K + 1, XS = NN * NP, XC = 3 * XS;
  extern __shared__ double sm[];  // [cpb][3][NN][NP]
  const int tid = threadIdx.x, l = tid / NP, col = tid - l * NP;
  const int c0 = blockIdx.x * cpb, cnt = min(cpb, mesh.nc - c0);
  rhs_rows<K, 2, NP, 3>(sm, XC, rho, u, nullptr, c0, cnt);
  __syncthreads();
  if (l < cnt) {
    const long c = c0 + l;
    if (mesh.dts) wgrav *= mesh.dts[c];  // per-member time step
    double *x = sm + l * XC + col;
    double r[NP], ux[NP], uz[NP], a[NN];
    rhs_col<K, 2>(x, r);
    rhs_col<K, 2>(x + XS, ux);
    rhs_col<K, 2>(x + 2 * XS, uz);
    const double *jw = mesh.jw + c * mesh.jw_stride + col;
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      const double t = fma(0.5 * M2, fma(ux[q], ux[q], uz[q] * uz[q]), wgrav * uz[q]);
      r[q] = -t * r[q] * __ldg(jw + q * NP);
    }
    eo_integ<K, 2, NP, true, false>(r, r, a);
#pragma unroll
    for (int i = 0; i < NN; ++i) x[i * NP] = a[i];
  }
  __syncthreads();
  for (int e = tid; e < cnt * NN; e += blockDim.x) {
    const int lo = e / NN, iz = e - lo * NN;
    double a[NP], out[NN];
#pragma unroll
    for (int q = 0; q < NP; ++q) a[q] = sm[lo * XC + iz * NP + q];
    eo_integ<K, 2, NP, true, false>(a, a, out);
    const long g = ((long)(c0 + lo) * NN + iz) * NN;
#pragma unroll
    for (int q = 0; q < NN; ++q) dst[g + q] = base[g + q] + out[q];
  }
}

// ============================================================ launchers ===
inline void rhs_sources(SrcPtrs &sp, int &nsrc, int kind, int stage, const double *const *src) {
  const int nsrc_tab[3][3] = {{2, 4, 6}, {4, 7, 9}, {5, 8, 11}};
  nsrc = nsrc_tab[kind][stage - 1];
  for (int i = 0; i < nsrc; ++i) sp.p[i] = src[i];
}

// Meshes below this many cells integrate faces point by point.  The second
// stage's three right-hand sides, a face per thread / a point per thread:
// 231 / 158 us at 800 cells, k = 4; 182 / 146 at 2304, k = 3; 554 / 535 at 4140,
// k = 5; 197 / 207 at 8192, k = 2; 554 / 561 at 8192, k = 4.  With hanging faces,
// which are of either parity, a mesh has more faces per cell and a thread more
// registers: third stage at k = 3, 788 / 638 us at 9120 cells, 1300 / 1345 at
// 22000; at k = 5 1792 / 1540 and 3256 / 3480.
constexpr int RHS_POINT_CELLS = 6000, RHS_POINT_CELLS_HANG = 12000;
template <int K, int KIND, bool HG>
int rhs_face_launch(const atm_ctx &c, int stage, double *dst, int way, const SrcPtrs &sp,
                    const StageCoef &co) {
  const int per = way == FACE_HELD ? 2 : 1;  // as way_faces
  // even faces: the momentum walls, and hanging faces
  const long n = (long)c.nc * per * (HG || KIND == 1 ? 2 : 1);
  if (c.nc < (HG ? RHS_POINT_CELLS_HANG : RHS_POINT_CELLS)) {
    // odd faces; even walls of the momentum equation; hanging faces
    const long m = (long)c.nc * per * (1 + (KIND == 1 ? 1 : 0) + (HG ? 2 : 0));
    void (*fp)(double *, int, SrcPtrs, StageCoef, Mesh) =
        stage == 1 ? k_rhs_face_points<K, 1, KIND, HG>
                   : (stage == 2 ? k_rhs_face_points<K, 2, KIND, HG>
                                 : k_rhs_face_points<K, 3, KIND, HG>);
    fp<<<(unsigned)((m + RHS_FPB - 1) / RHS_FPB), RHS_FPB * (2 * K + 1), 0, c.stream>>>(
        dst, way, sp, co, c.mesh);
    ATM_CHECK_LAUNCH("k_rhs_face_points");
    return ATM_OK;
  }
  void (*fn)(double *, int, SrcPtrs, StageCoef, Mesh) =
      stage == 1 ? k_rhs_face<K, 1, KIND, HG>
                 : (stage == 2 ? k_rhs_face<K, 2, KIND, HG> : k_rhs_face<K, 3, KIND, HG>);
  fn<<<(unsigned)((n + 63) / 64), 64, 0, c.stream>>>(dst, way, sp, co, c.mesh);
  ATM_CHECK_LAUNCH("k_rhs_face");
  return ATM_OK;
}

template <int KIND, bool HG>
int rhs_face_dispatch(const atm_ctx &c, int stage, double *dst, int way, const SrcPtrs &sp,
                      const StageCoef &co) {
  ATM_DISPATCH_K(c.k, (rhs_face_launch<K, KIND, HG>(c, stage, dst, way, sp, co)));
}

}  // namespace atm
