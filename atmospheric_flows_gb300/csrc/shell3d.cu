// The reference's own test case in 3D: FE_DGQ(1) hexahedra on a spherical
// shell with radial gravity (Atmospheric_Flow.cc:279-286, euler_operator.h,
// dim = 3, degree 1, QGauss(3)).  One kernel family restates every operator
// of the IMEX step for this case, and a host time loop drives it exactly as
// the 2D path does (Atmospheric_Flow.cc:1100-1257).
//
// Layout: scalar fields [cell][8], velocity [cell][3][8]; node v = ix + 2 iy
// + 4 iz on the cell's vertices (Gauss-Lobatto points of degree 1).  Cell
// geometry at the 27 Gauss points: dxi_e/dx_i * JxW (9 values), JxW, and the
// gravity direction e_r a^2/r^2 (3); face geometry at the 9 points of each
// local face: outward normal (3) and JxW.  The face-point permutation handles
// the rotated and flipped parameterisations where cubed-sphere patches meet.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <vector>

#include "atm_device.cuh"

struct atm3_ctx;

namespace atm {
namespace s3 {

constexpr int NN = 8, NQ = 27, NF = 9;
constexpr double EARTH_A = 6.37122e6;  // equation_data.h:26

__constant__ double c_phi[NQ][NN];      // basis values at the cell points
__constant__ double c_dphi[NQ][NN][3];  // reference derivatives at the cell points
__constant__ double c_fphi[6][NF][NN];  // basis values at the face points
__constant__ double c_psi[NF][4];       // bilinear basis at the face points (any face)
__constant__ double c_line[2];          // 1 - g_0 and g_0 of the three-point rule

struct Geo3 {
  int nc;
  const double *cg;    // [nc][27][13]: G[e][i] (9), JxW, gvec (3)
  const double *fg;    // [nc][6][9][4]: n (3), JxW
  const int *nbr;      // [nc][6]: neighbour or -1 (wall)
  const int *nbf;      // [nc][6]: neighbour's local face
  const int *nperm;    // [nc][6][9]: neighbour's point of each own face point
  int nfaces = 0;      // faces in `own`
  const int *own;      // cell * 6 + face of every face's owner: the inner faces, then the walls
};

struct Coef3 {
  double ca[3], ct[3], cg[3];
  int nst, ng;
  double dt, Ma, Fr;
};

__device__ __forceinline__ void load8(const double *v, int c, int ncomp, int comp, double *t) {
  const double *s = v + ((long)c * ncomp + comp) * NN;
#pragma unroll
  for (int i = 0; i < NN; ++i) t[i] = s[i];
}
__device__ __forceinline__ double at_q(const double *t, int q) {
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < NN; ++i) s = fma(c_phi[q][i], t[i], s);
  return s;
}
// k-th (k < 4) vertex of local face f, in increasing vertex order: the
// vertices whose bit f/2 equals f%2.  The other four basis functions vanish
// on the face exactly.
__device__ __forceinline__ int fnode(int f, int k) {
  const int a = f >> 1, lo = k & ((1 << a) - 1);
  return lo | ((f & 1) << a) | ((k >> a) << (a + 1));
}

// The kernels below are bound by their FP64 instructions (two lanes per clock
// and SM; an instruction costs the same with few active lanes as with 32), so
// their tasks are dealt out over all threads of a block and every quantity is
// computed once:
//   * a face is integrated once, by its owner (the "+" side of the face list),
//     and its nodal integrals are stored for both cells.  On a face the four
//     basis functions are the bilinear ones, the same table for every face;
//     the neighbour's point and basis row come from the face's permutation;
//   * a field is interpolated along x on the four edges first, then at each
//     point by the bilinear weights of the other two directions (5 instead of 8
//     FMAs a point), and cell integrals contract z, y, x in turn (372 instead
//     of 864 FMAs per component; the derivative of the degree-1 basis is -1, +1);
//   * what is linear with fixed coefficients is a dense table: B of the cell's
//     own and its neighbours' vertices (20 FMAs per output), D, and the volume
//     part of C for the current p_fix.
// Measured on GB300 at 6144 cells against a warp per cell with every face from
// both sides and dense point sums: B with A^{-1} 94 -> 15 us, C/D 99 -> 35 us
// (25 of them the faces), the second stage's three right-hand sides together
// 865 -> 335 us; the FP64 pipe is 64-84% busy.
constexpr int FPB = 32;  // faces per block of the face kernels, 9 threads each

// interpolation of degree-1 values to the three points, and its transpose
__device__ __forceinline__ void line3(double a, double b, double s, double t, double (&v)[3]) {
  v[0] = fma(s, a, t * b);  // s = 1 - g_0, t = g_0 (g_2 = 1 - g_0)
  v[1] = 0.5 * (a + b);
  v[2] = fma(t, a, s * b);
}
__device__ __forceinline__ void line3_t(double v0, double v1, double v2, double s, double t,
                                        double &a, double &b) {
  const double h = 0.5 * v1;
  a = fma(s, v0, fma(t, v2, h));
  b = fma(t, v0, fma(s, v2, h));
}

// ---------------------------------------------------------- face tables --
// A face kernel's view of one face point: own cell and face, neighbour (-1: a
// wall), the two bilinear rows and the normal times the face weight
struct FacePt {
  int c, f, nb, nf;
  double w[4], v[4], n[3];
};
__device__ __forceinline__ FacePt face_point(const Geo3 &g, int e, int q) {
  FacePt P;
  P.c = e / 6;
  P.f = e - P.c * 6;
  P.nb = g.nbr[e];
  P.nf = g.nbf[e];
  const int qn = g.nperm[e * NF + q];
  const double *fq = g.fg + ((long)e * NF + q) * 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    P.w[k] = c_psi[q][k];
    P.v[k] = c_psi[qn][k];
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) P.n[d] = fq[d] * fq[3];
  return P;
}
// traces of component comp of a field with ncomp components
__device__ __forceinline__ double own_tr(const FacePt &P, const double *v, int ncomp, int comp) {
  const double *s = v + ((long)P.c * ncomp + comp) * NN;
  double r = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) r = fma(P.w[k], __ldg(s + fnode(P.f, k)), r);
  return r;
}
__device__ __forceinline__ double nb_tr(const FacePt &P, const double *v, int ncomp, int comp) {
  const double *s = v + ((long)P.nb * ncomp + comp) * NN;
  double r = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) r = fma(P.v[k], __ldg(s + fnode(P.nf, k)), r);
  return r;
}
// nodal integrals of the block's face values F[face][comp][9]: minus for the
// owner, plus for the neighbour, Fb[cell][face][comp][4]
template <int NC>
__device__ __forceinline__ void face_store(const double *F, const Geo3 &g, int f0, int nf,
                                           double *__restrict__ Fb) {
  for (int t = threadIdx.x; t < nf * 2 * NC * 4; t += blockDim.x) {
    const int lf = t / (8 * NC), r = t - lf * 8 * NC, side = r / (4 * NC);
    const int comp = (r - side * 4 * NC) >> 2, k = r & 3;
    const int e = g.own[f0 + lf], nb = g.nbr[e];
    if (side && nb < 0) continue;
    const double *v = F + (lf * NC + comp) * NF;
    double o = 0.0;
#pragma unroll
    for (int q = 0; q < NF; ++q)
      o = fma(c_psi[side ? g.nperm[e * NF + q] : q][k], v[q], o);
    const long to = side ? (long)nb * 6 + g.nbf[e] : e;
    Fb[(to * NC + comp) * 4 + k] = side ? o : -o;
  }
}

// ------------------------------------------------- explicit rhs, faces --
// KIND 0 density (euler_operator.h:478-692, no boundary term), 1 momentum
// (:1891-2305, walls with p_D = p), 2 energy (:1012-1361, the stage-2 kinetic
// jump mixing in u_old :1182-1183 and the stage-3 total rho E jump
// :1290-1336; the division by rho in the reference's E cancels).
// src = (rho, u, [p])^(j) for j < nst.
template <int KIND>
__global__ void __launch_bounds__(NF * FPB, 2)
    k3_rhs_face(double *__restrict__ Fb, SrcPtrs src, Coef3 co, int hstage, Geo3 g) {
  constexpr int NC = KIND == 1 ? 3 : 1, PER = KIND == 0 ? 2 : 3;
  constexpr double ig = 1.0 / (GAS_GAMMA - 1.0), hgf = GAS_GAMMA * ig;
  __shared__ double sF[FPB][NC][NF];
  const int f0 = blockIdx.x * FPB, nf = min(FPB, g.nfaces - f0);
  const int lf = threadIdx.x / NF, q = threadIdx.x - lf * NF;
  if (lf < nf) {
    const FacePt P = face_point(g, g.own[f0 + lf], q);
    double F[NC];
#pragma unroll
    for (int d = 0; d < NC; ++d) F[d] = 0.0;
    double xo[3], xn[3];  // state 0's velocity traces (stage 2, energy)
    if (P.nb < 0) {
      if constexpr (KIND == 1)
        for (int j = 0; j < co.nst; ++j) {
          const double w = co.ct[j] * co.dt / (co.Ma * co.Ma) * own_tr(P, src.p[PER * j + 2], 1, 0);
#pragma unroll
          for (int d = 0; d < 3; ++d) F[d] = fma(w, P.n[d], F[d]);
        }
    } else {
      for (int j = 0; j < co.nst; ++j) {
        const double ro = own_tr(P, src.p[PER * j], 1, 0), rn = nb_tr(P, src.p[PER * j], 1, 0);
        double uo[3], un[3], a = 0.0, b = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          uo[d] = own_tr(P, src.p[PER * j + 1], 3, d);
          un[d] = nb_tr(P, src.p[PER * j + 1], 3, d);
          a = fma(uo[d], P.n[d], a);
          b = fma(un[d], P.n[d], b);
        }
        const double lam = abs_max(a, b), wa = co.ca[j] * co.dt;
        if constexpr (KIND == 0) {
          F[0] = fma(0.5 * wa, fma(lam, ro - rn, fma(ro, a, rn * b)), F[0]);
        } else {
          const double po = own_tr(P, src.p[PER * j + 2], 1, 0);
          const double pn = nb_tr(P, src.p[PER * j + 2], 1, 0);
          if constexpr (KIND == 1) {
            const double ps = 0.5 * co.ct[j] * co.dt / (co.Ma * co.Ma) * (po + pn);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const double mo = ro * uo[d], mn = rn * un[d];
              const double t = fma(lam, mo - mn, fma(mo, a, mn * b));
              F[d] = fma(0.5 * wa, t, fma(ps, P.n[d], F[d]));
            }
          } else {
            // per side: k rho |u|^2 + k2 p over the flux, + k3 p in the jump
            const double we = hstage == 3 ? wa : co.ct[j] * co.dt;
            const double k1 = 0.25 * wa * co.Ma * co.Ma, k2 = 0.5 * hgf * we, k3 = 0.5 * ig * we;
            double so = 0.0, sn = 0.0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              so = fma(uo[d], uo[d], so);
              sn = fma(un[d], un[d], sn);
            }
            const double ko = k1 * ro * so, kn = k1 * rn * sn;
            double jo = ko, jn = kn;
            if (hstage == 2) {
              if (j == 0) {
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                  xo[d] = uo[d];
                  xn[d] = un[d];
                }
              } else {
                so = sn = 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                  so = fma(uo[d], xo[d], so);
                  sn = fma(un[d], xn[d], sn);
                }
                jo = k1 * ro * so;
                jn = k1 * rn * sn;
              }
            }
            F[0] = fma(fma(k2, po, ko), a, F[0]);
            F[0] = fma(fma(k2, pn, kn), b, F[0]);
            F[0] = fma(lam, fma(k3, po, jo) - fma(k3, pn, jn), F[0]);
          }
        }
      }
    }
#pragma unroll
    for (int d = 0; d < NC; ++d) sF[lf][d][q] = F[d];
  }
  __syncthreads();
  face_store<NC>(&sF[0][0][0], g, f0, nf, Fb);
}

// -------------------------------------------------- explicit rhs, cells --
// euler_operator.h:344-473 (density), 1622-1886 (momentum), 745-1007 (energy,
// with the radial gravity work :790-811), plus the face integrals Fb.
// `cpb` cells per block, 27 threads each.  `fields` counts the scalar fields
// that the block interpolates: (rho, u, [p])^(j), then KIND 1: the density
// being solved for (stages 1, 2), KIND 2: the kinetic (rho, u).
template <int KIND>
__global__ void __launch_bounds__(27 * 14)
    k3_rhs_cell(double *__restrict__ dst, SrcPtrs src, Coef3 co, int hstage, int fields, Geo3 g,
                const double *__restrict__ Fb, int cpb) {
  constexpr int NC = KIND == 1 ? 3 : 1, PER = KIND == 0 ? 2 : 3, SF = KIND == 0 ? 4 : 5;
  constexpr double ig = 1.0 / (GAS_GAMMA - 1.0), hgf = GAS_GAMMA * ig;
  extern __shared__ double sm[];  // [cpb][fields][4][3], then [cpb][NC][4][27]
  __shared__ double spsi[NF][4];
  const int per = max(fields * 12, NC * 4 * NQ);
  const int c0 = blockIdx.x * cpb, cnt = min(cpb, g.nc - c0);
  const double s = c_line[0], t = c_line[1];
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < NF * 4; e += nt) spsi[e >> 2][e & 3] = c_psi[e >> 2][e & 3];
  // x-lines: (cell, field, edge)
  for (int e = tid; e < cnt * fields * 4; e += nt) {
    const int l = e / (fields * 4), r = e - l * fields * 4, fd = r >> 2, m = r & 3;
    const long c = c0 + l;
    const int j = fd / SF, k = fd - j * SF;  // state and its field
    const double *v;
    if (j < co.nst) {
      v = k == 0 ? src.p[PER * j] + c * NN
                 : k < 4 ? src.p[PER * j + 1] + (c * 3 + k - 1) * NN : src.p[PER * j + 2] + c * NN;
    } else {
      v = k == 0 ? src.p[PER * co.nst] + c * NN : src.p[PER * co.nst + 1] + (c * 3 + k - 1) * NN;
    }
    double o[3];
    line3(__ldg(v + 2 * m), __ldg(v + 2 * m + 1), s, t, o);
#pragma unroll
    for (int i = 0; i < 3; ++i) sm[l * per + r * 3 + i] = o[i];
  }
  __syncthreads();
  const int l = tid / NQ, q = tid - l * NQ;
  double V[NC], G[NC][3];
  if (l < cnt) {
    const double *X = sm + l * per + q % 3;
    double w[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) w[m] = spsi[q / 3][m];
    const double *cq = g.cg + ((long)(c0 + l) * NQ + q) * 13;
    auto val = [&](int fd) {
      double r = 0.0;
#pragma unroll
      for (int m = 0; m < 4; ++m) r = fma(w[m], X[(fd * 4 + m) * 3], r);
      return r;
    };
    double P[NC][3], gr = 0.0;  // physical fluxes; gravity's density / work
#pragma unroll
    for (int d = 0; d < NC; ++d) {
      V[d] = 0.0;
#pragma unroll
      for (int i = 0; i < 3; ++i) P[d][i] = 0.0;
    }
    for (int j = 0; j < co.nst; ++j) {
      const double r = val(SF * j), wa = co.ca[j] * co.dt;
      double u[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) u[d] = val(SF * j + 1 + d);
      if constexpr (KIND == 0) {
        if (j == 0) V[0] = r;
        const double wr = wa * r;
#pragma unroll
        for (int i = 0; i < 3; ++i) P[0][i] = fma(wr, u[i], P[0][i]);
      } else if constexpr (KIND == 1) {
        const double pp = co.ct[j] * co.dt / (co.Ma * co.Ma) * val(SF * j + 4);
        gr = fma(co.cg[j], r, gr);
        const double wr = wa * r;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if (j == 0) V[d] = r * u[d];
          const double ru = wr * u[d];
#pragma unroll
          for (int i = d; i < 3; ++i) P[d][i] = fma(ru, u[i], P[d][i]);  // symmetric
          P[d][d] += pp;
        }
      } else {
        const double p = val(SF * j + 4), M2 = co.Ma * co.Ma;
        const double k = r * fma(u[0], u[0], fma(u[1], u[1], u[2] * u[2]));
        if (j == 0) V[0] = fma(ig, p, 0.5 * M2 * k);  // rho E
        const double ug = fma(u[0], cq[10], fma(u[1], cq[11], u[2] * cq[12]));
        gr = fma(co.cg[j] * r, ug, gr);
        const double h = fma(0.5 * wa * M2, k, co.ct[j] * co.dt * hgf * p);
#pragma unroll
        for (int i = 0; i < 3; ++i) P[0][i] = fma(h, u[i], P[0][i]);
      }
    }
    if constexpr (KIND == 1) {
      if (fields > SF * co.nst) gr = fma(co.cg[co.nst], val(SF * co.nst), gr);
      const double wg = co.dt / (co.Fr * co.Fr) * gr;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        V[d] = fma(-wg, cq[10 + d], V[d]);
#pragma unroll
        for (int i = 0; i < d; ++i) P[d][i] = P[i][d];
      }
    }
    if constexpr (KIND == 2) {
      const double M2 = co.Ma * co.Ma, r = val(SF * co.nst);
      double u[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) u[d] = val(SF * co.nst + 1 + d);
      if (hstage < 3) {  // gravity work of the density being solved for
        const double ug = fma(u[0], cq[10], fma(u[1], cq[11], u[2] * cq[12]));
        gr = fma(co.cg[co.nst] * r, ug, gr);
      }
      V[0] = fma(-0.5 * M2 * r, fma(u[0], u[0], fma(u[1], u[1], u[2] * u[2])), V[0]);
      V[0] = fma(-co.dt * M2 / (co.Fr * co.Fr), gr, V[0]);
    }
#pragma unroll
    for (int d = 0; d < NC; ++d) {
      V[d] *= cq[9];
#pragma unroll
      for (int e = 0; e < 3; ++e)
        G[d][e] = fma(cq[3 * e], P[d][0], fma(cq[3 * e + 1], P[d][1], cq[3 * e + 2] * P[d][2]));
    }
  }
  __syncthreads();
  if (l < cnt) {
    double *o = sm + l * per + q;
#pragma unroll
    for (int d = 0; d < NC; ++d) {
      o[(d * 4) * NQ] = V[d];
#pragma unroll
      for (int e = 0; e < 3; ++e) o[(d * 4 + 1 + e) * NQ] = G[d][e];
    }
  }
  __syncthreads();
  // z, then y, then x: each task replaces its own line's values
  for (int e = tid; e < cnt * NC * 9; e += nt) {
    const int lo = e / (NC * 9), r = e - lo * NC * 9, d = r / 9;
    double *v = sm + lo * per + d * 4 * NQ + (r - d * 9);
    double a, b;
    double *gz = v + 3 * NQ;
    const double z = gz[0] + gz[9] + gz[18];
    line3_t(v[0], v[9], v[18], s, t, a, b);
    v[0] = a - z;
    v[9] = b + z;
#pragma unroll
    for (int k = 1; k < 3; ++k) {
      double *y = v + k * NQ;
      line3_t(y[0], y[9], y[18], s, t, a, b);
      y[0] = a;
      y[9] = b;
    }
  }
  __syncthreads();
  for (int e = tid; e < cnt * NC * 6; e += nt) {
    const int lo = e / (NC * 6), r = e - lo * NC * 6, d = r / 6, k = r - d * 6;
    double *v = sm + lo * per + d * 4 * NQ + (k / 3) * 9 + k % 3;
    double a, b;
    const double *gy = v + 2 * NQ;
    const double y = gy[0] + gy[3] + gy[6];
    line3_t(v[0], v[3], v[6], s, t, a, b);
    v[0] = a - y;
    v[3] = b + y;
    double *gx = v + NQ;
    line3_t(gx[0], gx[3], gx[6], s, t, a, b);
    gx[0] = a;
    gx[3] = b;
  }
  __syncthreads();
  for (int e = tid; e < cnt * NC * 4; e += nt) {
    const int lo = e / (NC * 4), r = e - lo * NC * 4, d = r >> 2, y = r & 1, z = (r >> 1) & 1;
    const double *v = sm + lo * per + d * 4 * NQ + z * 9 + y * 3;
    double a, b;
    const double x = v[NQ] + v[NQ + 1] + v[NQ + 2];
    line3_t(v[0], v[1], v[2], s, t, a, b);
    const long c = c0 + lo;
    const double *F = Fb + (c * 6 * NC + d) * 4;  // face f at f * NC * 4
    // vertex (x, y, z): faces x, 2 + y, 4 + z
    const double *Fy = F + (2 + y) * NC * 4 + 2 * z, *Fz = F + (4 + z) * NC * 4 + 2 * y;
    double *o = dst + (c * 3 * (NC == 3) + c * (NC == 1) + d) * NN + 2 * y + 4 * z;
    o[0] = (a - x) + F[y + 2 * z] + Fy[0] + Fz[0];
    o[1] = (b + x) + F[NC * 4 + y + 2 * z] + Fy[1] + Fz[1];
  }
}

// ------------------------------------------------------------ B and D tables --
// wb [nc][8][24]: B of the cell's own values, output (d, i) from vertex j:
//   -sum_q phi_j G[.][d] . grad phi_i + half the face terms (walls: all of it)
// nb [nc][12][24]: of the neighbours', output (d, i) from vertex k' of the face
// along axis a that holds i (row a * 4 + k'); dm [nc][8][8]: D.
__global__ void k3_tables(double *__restrict__ wb, double *__restrict__ nbt,
                          double *__restrict__ dm, Geo3 g) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)g.nc * 24) return;
  const int c = (int)(t / 24), o = (int)(t - (long)c * 24), d = o / NN, i = o - d * NN;
  double W[NN], D[NN];
  for (int j = 0; j < NN; ++j) W[j] = D[j] = 0.0;
  for (int q = 0; q < NQ; ++q) {
    const double *cq = g.cg + ((long)c * NQ + q) * 13;
    const double s = -(cq[d] * c_dphi[q][i][0] + cq[3 + d] * c_dphi[q][i][1] +
                       cq[6 + d] * c_dphi[q][i][2]);
    const double m = c_phi[q][i] * cq[9] / (GAS_GAMMA - 1.0);
    for (int j = 0; j < NN; ++j) {
      W[j] = fma(s, c_phi[q][j], W[j]);
      D[j] = fma(m, c_phi[q][j], D[j]);
    }
  }
  for (int a = 0; a < 3; ++a) {
    const int f = 2 * a + ((i >> a) & 1), e = c * 6 + f, nb = g.nbr[e];
    double N[4] = {0, 0, 0, 0};
    for (int q = 0; q < NF; ++q) {
      const double *fq = g.fg + ((long)e * NF + q) * 4;
      const double s = c_fphi[f][q][i] * fq[d] * fq[3] * (nb < 0 ? 1.0 : 0.5);
      for (int k = 0; k < 4; ++k) {
        const int j = fnode(f, k);
        W[j] = fma(s, c_fphi[f][q][j], W[j]);
        if (nb >= 0) N[k] = fma(s, c_psi[g.nperm[e * NF + q]][k], N[k]);
      }
    }
    for (int k = 0; k < 4; ++k) nbt[((long)c * 12 + a * 4 + k) * 24 + o] = N[k];
  }
  for (int j = 0; j < NN; ++j) {
    wb[((long)c * NN + j) * 24 + o] = W[j];
    if (d == 0) dm[((long)c * NN + j) * NN + i] = D[j];
  }
}

// ------------------------------------------------------------------- B --
// euler_operator.h:1512-1617; mode 0 dst = cB B p, 1 dst -= cB B p,
// 2 dst = cB A^{-1} B p.  24 threads per cell, one per output.
constexpr int CB_B = 8;
__global__ void __launch_bounds__(24 * CB_B)
    k3_B(double *__restrict__ dst, const double *__restrict__ p, double cB,
         const double *__restrict__ ainv, int mode, const double *__restrict__ wb,
         const double *__restrict__ nbt, Geo3 g) {
  __shared__ double so[CB_B][NN], sn[CB_B][24], sb[CB_B][24];
  const int l = threadIdx.x / 24, o = threadIdx.x - l * 24;
  const int c = blockIdx.x * CB_B + l;
  const bool active = c < g.nc;
  if (active) {
    const int f = o >> 2, nb = g.nbr[c * 6 + f];  // vertex o & 3 of the neighbour across f
    sn[l][o] = nb < 0 ? 0.0 : __ldg(p + (long)nb * NN + fnode(g.nbf[c * 6 + f], o & 3));
    if (o < NN) so[l][o] = __ldg(p + (long)c * NN + o);
  }
  __syncthreads();
  const int d = o / NN, i = o - d * NN;
  const long gi = (long)c * 24 + o;
  double r = 0.0;
  if (active) {
    const double *W = wb + (long)c * NN * 24 + o, *N = nbt + (long)c * 12 * 24 + o;
#pragma unroll
    for (int j = 0; j < NN; ++j) r = fma(__ldg(W + j * 24), so[l][j], r);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double *v = sn[l] + (2 * a + ((i >> a) & 1)) * 4;
#pragma unroll
      for (int k = 0; k < 4; ++k) r = fma(__ldg(N + (a * 4 + k) * 24), v[k], r);
    }
    r *= cB;
    if (mode == 0) dst[gi] = r;
    else if (mode == 1) dst[gi] -= r;
    sb[l][o] = r;
  }
  if (mode != 2) return;  // uniform over the grid
  __syncthreads();
  if (active) {
    const double *A = ainv + (long)c * NN * NN + i;  // symmetric
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < NN; ++j) s = fma(__ldg(A + j * NN), sb[l][d * NN + j], s);
    dst[gi] = s;
  }
}

// ----------------------------------------------------------------- C/D --
// euler_operator.h:1386-1507
// cm [nc][24][8]: minus the volume part of C for the frozen p_fix, output i from
// w's (d, j): gamma/(gamma-1) sum_q p_fix phi_j G[.][d] . grad phi_i.
// 24 threads per cell: (d, i), all j.
__global__ void __launch_bounds__(192)
    k3_prep_C(double *__restrict__ cm, const double *__restrict__ pfix, Geo3 g) {
  constexpr double hgf = GAS_GAMMA / (GAS_GAMMA - 1.0);
  __shared__ double sphi[NQ][NN], sd[NQ][NN][3], spf[8][NQ];
  for (int e = threadIdx.x; e < NQ * NN; e += blockDim.x) {
    sphi[e / NN][e % NN] = c_phi[e / NN][e % NN];
    for (int k = 0; k < 3; ++k) sd[e / NN][e % NN][k] = c_dphi[e / NN][e % NN][k];
  }
  __syncthreads();
  const int c0 = blockIdx.x * 8, cnt = min(8, g.nc - c0);
  for (int e = threadIdx.x; e < cnt * NQ; e += blockDim.x) {
    const int l = e / NQ, q = e - l * NQ;
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < NN; ++j) s = fma(sphi[q][j], __ldg(pfix + (long)(c0 + l) * NN + j), s);
    spf[l][q] = hgf * s;
  }
  __syncthreads();
  const int l = threadIdx.x / 24, o = threadIdx.x - l * 24, d = o / NN, i = o - d * NN;
  if (l >= cnt) return;
  double W[NN];
#pragma unroll
  for (int j = 0; j < NN; ++j) W[j] = 0.0;
  for (int q = 0; q < NQ; ++q) {
    const double *cq = g.cg + ((long)(c0 + l) * NQ + q) * 13;
    const double s = spf[l][q] * fma(__ldg(cq + d), sd[q][i][0],
                                     fma(__ldg(cq + 3 + d), sd[q][i][1], __ldg(cq + 6 + d) * sd[q][i][2]));
#pragma unroll
    for (int j = 0; j < NN; ++j) W[j] = fma(s, sphi[q][j], W[j]);
  }
  double *out = cm + ((long)(c0 + l) * 24 + d * NN) * NN + i;
#pragma unroll
  for (int j = 0; j < NN; ++j) out[j * NN] = W[j];
}
// face part of C: minus its nodal integrals, Fb[cell][face][4]
__global__ void __launch_bounds__(NF * FPB)
    k3_face_C(double *__restrict__ Fb, const double *__restrict__ w,
              const double *__restrict__ pfix, Geo3 g) {
  constexpr double ig = 1.0 / (GAS_GAMMA - 1.0), hgf = GAS_GAMMA * ig;
  __shared__ double sF[FPB][1][NF];
  const int f0 = blockIdx.x * FPB, nf = min(FPB, g.nfaces - f0);
  const int lf = threadIdx.x / NF, q = threadIdx.x - lf * NF;
  if (lf < nf) {
    const FacePt P = face_point(g, g.own[f0 + lf], q);
    double F = 0.0;
    if (P.nb >= 0) {  // no boundary term
      const double po = own_tr(P, pfix, 1, 0), pn = nb_tr(P, pfix, 1, 0);
      double a = 0.0, b = 0.0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        a = fma(own_tr(P, w, 3, d), P.n[d], a);
        b = fma(nb_tr(P, w, 3, d), P.n[d], b);
      }
      F = fma(0.5 * ig * abs_max(a, b), po - pn, 0.5 * hgf * fma(po, a, pn * b));
    }
    sF[lf][0][q] = F;
  }
  __syncthreads();
  face_store<1>(&sF[0][0][0], g, f0, nf, Fb);
}
// mode 0 dst = cC C w; 1 dst = D p - cC C w; 2 dst = invd .* (D p - cC C w);
// 3 dst -= cC C w.  A warp per cell: lane (part, i), part 0..2 the component of
// w, part 3 p; two shuffles add the parts.
constexpr int CB_CD = 8;
__global__ void __launch_bounds__(32 * CB_CD)
    k3_CD(double *__restrict__ dst, const double *__restrict__ w, const double *__restrict__ p,
          double cC, const double *__restrict__ invd, int mode, const double *__restrict__ cm,
          const double *__restrict__ dm, const double *__restrict__ Fb, Geo3 g) {
  const int l = threadIdx.x >> 5, lane = threadIdx.x & 31, part = lane >> 3, i = lane & 7;
  const int c = blockIdx.x * CB_CD + l;
  if (c >= g.nc) return;  // warp-uniform
  const bool withD = mode == 1 || mode == 2;
  double in = 0.0;  // this lane's input value (part, vertex i)
  if (part < 3) in = cC * __ldg(w + (long)c * 24 + lane);
  else if (withD) in = __ldg(p + (long)c * NN + i);
  const double *M = part < 3 ? cm + ((long)c * 24 + part * NN) * NN + i : dm + (long)c * NN * NN + i;
  double o = 0.0;
#pragma unroll
  for (int j = 0; j < NN; ++j)
    o = fma(__ldg(M + j * NN), __shfl_sync(0xffffffffu, in, (part << 3) + j), o);
  o += __shfl_xor_sync(0xffffffffu, o, 8);
  o += __shfl_xor_sync(0xffffffffu, o, 16);
  if (lane >= NN) return;
  const double *F = Fb + (long)c * 24;
  const int x = i & 1, y = (i >> 1) & 1, z = i >> 2;
  o = fma(cC, F[x * 4 + y + 2 * z] + F[(2 + y) * 4 + x + 2 * z] + F[(4 + z) * 4 + x + 2 * y], o);
  const long gi = (long)c * NN + i;
  if (mode == 0) dst[gi] = -o;
  else if (mode == 1) dst[gi] = o;
  else if (mode == 2) dst[gi] = invd[gi] * o;
  else dst[gi] += o;
}

// ------------------------------------------------ cell-wise mass inverses --
// inv = (sum_q w(q) phi_i phi_j JxW)^{-1} per cell, weight tile or 1;
// Gauss-Jordan with partial pivoting on the 8x8 block
__global__ void k3_block_inverse(double *__restrict__ inv, const double *__restrict__ weight,
                                 Geo3 g) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.nc) return;
  double wt[NN];
  if (weight) load8(weight, c, 1, 0, wt);
  double M[NN][2 * NN];
  for (int i = 0; i < NN; ++i)
    for (int j = 0; j < 2 * NN; ++j) M[i][j] = (j - NN == i) ? 1.0 : 0.0;
  for (int q = 0; q < NQ; ++q) {
    const double jw = g.cg[((long)c * NQ + q) * 13 + 9] * (weight ? at_q(wt, q) : 1.0);
    for (int i = 0; i < NN; ++i)
      for (int j = 0; j < NN; ++j) M[i][j] += jw * c_phi[q][i] * c_phi[q][j];
  }
  for (int k = 0; k < NN; ++k) {
    int piv = k;
    for (int i = k + 1; i < NN; ++i)
      if (fabs(M[i][k]) > fabs(M[piv][k])) piv = i;
    if (piv != k)
      for (int j = 0; j < 2 * NN; ++j) { const double t = M[k][j]; M[k][j] = M[piv][j]; M[piv][j] = t; }
    const double d = 1.0 / M[k][k];
    for (int j = 0; j < 2 * NN; ++j) M[k][j] *= d;
    for (int i = 0; i < NN; ++i) {
      if (i == k) continue;
      const double f = M[i][k];
      for (int j = 0; j < 2 * NN; ++j) M[i][j] -= f * M[k][j];
    }
  }
  for (int i = 0; i < NN; ++i)
    for (int j = 0; j < NN; ++j) inv[(long)c * NN * NN + i * NN + j] = M[i][NN + j];
}

// dst = scale * inv src, ncomp components per cell
__global__ void k3_block_apply(double *__restrict__ dst, const double *__restrict__ src,
                               const double *__restrict__ inv, int ncomp, double scale, int nc) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const double *A = inv + (long)c * NN * NN;
  for (int d = 0; d < ncomp; ++d) {
    double t[NN];
    load8(src, c, ncomp, d, t);
    for (int i = 0; i < NN; ++i) {
      double s = 0.0;
      for (int j = 0; j < NN; ++j) s += A[i * NN + j] * t[j];
      dst[((long)c * ncomp + d) * NN + i] = scale * s;
    }
  }
}

// mass apply dst = M_w src (ncomp components, weight tile or constant)
__global__ void k3_mass(double *__restrict__ dst, const double *__restrict__ src, int ncomp,
                        const double *__restrict__ weight, double scale, Geo3 g) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.nc) return;
  double wt[NN];
  if (weight) load8(weight, c, 1, 0, wt);
  for (int d = 0; d < ncomp; ++d) {
    double t[NN], out[NN] = {0};
    load8(src, c, ncomp, d, t);
    for (int q = 0; q < NQ; ++q) {
      const double v = at_q(t, q) * (weight ? at_q(wt, q) : scale) *
                       g.cg[((long)c * NQ + q) * 13 + 9];
#pragma unroll
      for (int i = 0; i < NN; ++i) out[i] += v * c_phi[q][i];
    }
    for (int i = 0; i < NN; ++i) dst[((long)c * ncomp + d) * NN + i] = out[i];
  }
}

// inverse diagonal of D (the Schur Jacobi, euler_operator.h:2607-2611)
__global__ void k3_invdiag_D(double *__restrict__ out, Geo3 g) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.nc) return;
  for (int i = 0; i < NN; ++i) {
    double s = 0.0;
    for (int q = 0; q < NQ; ++q)
      s += c_phi[q][i] * c_phi[q][i] * g.cg[((long)c * NQ + q) * 13 + 9];
    out[(long)c * NN + i] = (GAS_GAMMA - 1.0) / s;
  }
}

}  // namespace s3
}  // namespace atm

// ============================================================================
// Host side: context, set-up, operators and the IMEX loop
// ============================================================================
using namespace atm;
using namespace atm::s3;

struct atm3_ctx {
  int device = 0, nc = 0;
  cudaStream_t stream = nullptr;
  Geo3 g{};
  double *cg = nullptr, *fg = nullptr;
  int *nbr = nullptr, *nbf = nullptr, *nperm = nullptr, *own = nullptr;
  double *wb = nullptr, *nbt = nullptr, *dm = nullptr;  // B and D tables (k3_tables)
  double *cm = nullptr;    // C's volume part for the frozen p_fix (k3_prep_C)
  // [nc][6][3][4] face integrals, from a face kernel to the cell kernel behind it.
  // Everything runs on the one stream; `pair` keeps host threads that share the
  // handle from launching between the two
  double *fbuf = nullptr;
  std::mutex pair;
  double dt = 1.0, Ma = 1.0, Fr = 1.0;
  int hstage = 1, nsstage = 1;
  Tableau tab;
  double *rho_fix = nullptr, *pres_fix = nullptr, *u_fix = nullptr;
  double *minv = nullptr, *ainv = nullptr, *invd = nullptr;
  double *wv1 = nullptr, *ws1 = nullptr, *ws2 = nullptr;
  double *red = nullptr, *red_out = nullptr, *h_red = nullptr, *dsmall = nullptr;
  double *krylov = nullptr;
  // solver
  bool solver = false;
  double eps = 1e-8;
  int max_its = 30000;
  bool scaled_tol = false, true_check = false;
  long steps = 0, picard_total = 0, krylov_total = 0, failures = 0;
  double *pool = nullptr;
  double *rho_old, *rho_2, *rho_3, *rho_cur, *rhs_rho, *p_old, *p_2, *p_3, *p_fix, *p_fix_old,
      *rhs_p, *u_old, *u_2, *u_3, *u_cur, *u_fixd, *rhs_u, *tmp_1;
  long ns() const { return (long)nc * NN; }
  long nv() const { return 3L * nc * NN; }
};

namespace {

constexpr int RESTART3 = 28;
#define TRY3(x)           \
  do {                    \
    int _rc = (x);        \
    if (_rc) return _rc;  \
  } while (0)

inline int blocks(int n) { return (n + 127) / 128; }

int upload_tables3() {
  // degree-1 basis on the vertices, 3-point Gauss rule on [0, 1]
  const double s = std::sqrt(0.6);
  const double gx[3] = {0.5 * (1.0 - s), 0.5, 0.5 * (1.0 + s)};
  double phi[NQ][NN], dphi[NQ][NN][3], fphi[6][NF][NN];
  auto q1 = [](const double xi[3], double *ph, double (*dp)[3]) {
    for (int v = 0; v < NN; ++v) {
      double f[3], df[3];
      for (int d = 0; d < 3; ++d) {
        const bool hi = (v >> d) & 1;
        f[d] = hi ? xi[d] : 1.0 - xi[d];
        df[d] = hi ? 1.0 : -1.0;
      }
      ph[v] = f[0] * f[1] * f[2];
      if (dp) {
        dp[v][0] = df[0] * f[1] * f[2];
        dp[v][1] = f[0] * df[1] * f[2];
        dp[v][2] = f[0] * f[1] * df[2];
      }
    }
  };
  for (int q = 0; q < NQ; ++q) {
    const double xi[3] = {gx[q % 3], gx[(q / 3) % 3], gx[q / 9]};
    q1(xi, phi[q], dphi[q]);
  }
  for (int f = 0; f < 6; ++f)
    for (int q = 0; q < NF; ++q) {
      const int d = f / 2, t0 = d == 0 ? 1 : 0, t1 = d == 2 ? 1 : 2;
      double xi[3];
      xi[d] = (double)(f % 2);
      xi[t0] = gx[q % 3];
      xi[t1] = gx[q / 3];
      q1(xi, fphi[f][q], nullptr);
    }
  double psi[NF][4];
  const double line[2] = {1.0 - gx[0], gx[0]};
  for (int q = 0; q < NF; ++q)
    for (int k = 0; k < 4; ++k)
      psi[q][k] = ((k & 1) ? gx[q % 3] : 1.0 - gx[q % 3]) * ((k >> 1) ? gx[q / 3] : 1.0 - gx[q / 3]);
  if (cudaMemcpyToSymbol(c_phi, phi, sizeof(phi)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_dphi, dphi, sizeof(dphi)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_fphi, fphi, sizeof(fphi)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_psi, psi, sizeof(psi)) != cudaSuccess ||
      cudaMemcpyToSymbol(c_line, line, sizeof(line)) != cudaSuccess) {
    set_error("failed to upload the 3D basis tables");
    return ATM_CUDA_ERROR;
  }
  return ATM_OK;
}

// x and dx/dxi of the degree-2 mapping of one cell at xi
void map3(const double *nodes, const double xi[3], double x[3], double J[3][3]) {
  double v[3][3], d[3][3];
  for (int e = 0; e < 3; ++e) {
    const double t = xi[e];
    v[e][0] = 2.0 * (t - 0.5) * (t - 1.0); v[e][1] = -4.0 * t * (t - 1.0); v[e][2] = 2.0 * t * (t - 0.5);
    d[e][0] = 4.0 * t - 3.0; d[e][1] = -8.0 * t + 4.0; d[e][2] = 4.0 * t - 1.0;
  }
  for (int i = 0; i < 3; ++i) {
    x[i] = 0.0;
    for (int e = 0; e < 3; ++e) J[i][e] = 0.0;
  }
  for (int c = 0; c < 3; ++c)
    for (int b = 0; b < 3; ++b)
      for (int a = 0; a < 3; ++a) {
        const double *X = nodes + 3 * ((c * 3 + b) * 3 + a);
        const double w = v[0][a] * v[1][b] * v[2][c];
        const double dw[3] = {d[0][a] * v[1][b] * v[2][c], v[0][a] * d[1][b] * v[2][c],
                              v[0][a] * v[1][b] * d[2][c]};
        for (int i = 0; i < 3; ++i) {
          x[i] += w * X[i];
          for (int e = 0; e < 3; ++e) J[i][e] += dw[e] * X[i];
        }
      }
}

// inverse of J (Ji[e][i] = dxi_e/dx_i) and det
double inv3(const double J[3][3], double Ji[3][3]) {
  const double det = J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) -
                     J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0]) +
                     J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
  for (int e = 0; e < 3; ++e)
    for (int i = 0; i < 3; ++i) {
      // cofactor of J[i][e]
      const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, e1 = (e + 1) % 3, e2 = (e + 2) % 3;
      Ji[e][i] = (J[i1][e1] * J[i2][e2] - J[i1][e2] * J[i2][e1]) / det;
    }
  return det;
}

int alloc3(atm3_ctx &c, double **p, size_t n) {
  ATM_CUDA(cudaMalloc(p, n * sizeof(double)));
  ATM_CUDA(cudaMemsetAsync(*p, 0, n * sizeof(double), c.stream));
  return ATM_OK;
}

void free3(atm3_ctx *c) {
  if (!c) return;
  double *ds[] = {c->cg, c->fg, c->rho_fix, c->pres_fix, c->u_fix, c->minv, c->ainv, c->invd,
                  c->wv1, c->ws1, c->ws2, c->red, c->red_out, c->dsmall, c->krylov, c->pool,
                  c->wb, c->nbt, c->dm, c->cm, c->fbuf};
  for (double *d : ds) cudaFree(d);
  cudaFree(c->nbr); cudaFree(c->nbf); cudaFree(c->nperm); cudaFree(c->own);
  if (c->h_red) cudaFreeHost(c->h_red);
  delete c;
}

int read3(atm3_ctx &c, const double *dev, int n) {
  ATM_CUDA(cudaMemcpyAsync(c.h_red, dev, n * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
  ATM_CUDA(cudaStreamSynchronize(c.stream));
  return ATM_OK;
}

Coef3 coef3(const atm3_ctx &c, int stage, bool rho_only) {
  Coef3 s{};
  const Tableau &t = c.tab;
  s.dt = c.dt; s.Ma = c.Ma; s.Fr = c.Fr;
  if (stage == 1) {
    s.nst = 1; s.ca[0] = t.a21; s.ct[0] = t.a21t;
    s.ng = 2; s.cg[0] = t.a21t; s.cg[1] = t.a22t;
  } else if (stage == 2) {
    s.nst = 2; s.ca[0] = t.a31; s.ca[1] = t.a32; s.ct[0] = t.a31t; s.ct[1] = t.a32t;
    s.ng = 3; s.cg[0] = t.a31t; s.cg[1] = t.a32t; s.cg[2] = t.a33t;
  } else {
    s.nst = 3; s.ca[0] = t.b1; s.ca[1] = t.b2; s.ca[2] = t.b3;
    s.ct[0] = t.b1; s.ct[1] = t.b2; s.ct[2] = t.b3;
    s.ng = 3; s.cg[0] = t.b1; s.cg[1] = t.b2; s.cg[2] = t.b3;
  }
  (void)rho_only;
  return s;
}
double icoef3(const atm3_ctx &c) { return c.hstage == 1 ? c.tab.a22t : c.tab.a33t; }

// ---- operators (positional source lists as the 2D entry points) -------------
inline int fblocks(const atm3_ctx &c) { return (c.g.nfaces + FPB - 1) / FPB; }
template <int KIND>
int rhs3(atm3_ctx &c, double *dst, const double *const *src) {
  const Coef3 co = coef3(c, c.hstage, KIND == 0);
  const int nsrc = KIND == 0 ? 2 * co.nst : KIND == 1 ? 3 * co.nst + (c.hstage < 3) : 3 * co.nst + 2;
  const int fields = KIND == 0 ? 4 * co.nst : KIND == 1 ? 5 * co.nst + (c.hstage < 3) : 5 * co.nst + 4;
  SrcPtrs sp{};
  for (int i = 0; i < nsrc; ++i) sp.p[i] = src[i];
  std::lock_guard<std::mutex> lock(c.pair);
  k3_rhs_face<KIND><<<fblocks(c), NF * FPB, 0, c.stream>>>(c.fbuf, sp, co, c.hstage, c.g);
  ATM_CHECK_LAUNCH("k3_rhs_face");
  // 14 cells: 378 of 384 threads; small shells take small blocks
  const int cpb = c.nc < 1500 ? 4 : 14, nc = KIND == 1 ? 3 : 1;
  const size_t sm = sizeof(double) * (size_t)cpb * std::max(fields * 12, nc * 4 * NQ);
  ATM_CUDA(allow_smem(k3_rhs_cell<KIND>, sm));
  k3_rhs_cell<KIND><<<(c.nc + cpb - 1) / cpb, NQ * cpb, sm, c.stream>>>(dst, sp, co, c.hstage, fields,
                                                                      c.g, c.fbuf, cpb);
  ATM_CHECK_LAUNCH("k3_rhs_cell");
  return ATM_OK;
}
int rhs_rho3(atm3_ctx &c, double *dst, const double *const *src) { return rhs3<0>(c, dst, src); }
// src: stage 1 {rho_old,u_old,p_old,rho_2}; 2 {.., u_2, p_2, rho_3};
// 3 {.., u_3, p_3}
int rhs_vel3(atm3_ctx &c, double *dst, const double *const *src) { return rhs3<1>(c, dst, src); }
// src: stage 1 {rho_old,u_old,p_old,rho_2,u_fix}; 2 {.., u_2, p_2, rho_3,
// u_fix}; 3 {.., u_3, p_3, rho_cur, u_cur}
int rhs_pres3(atm3_ctx &c, double *dst, const double *const *src) { return rhs3<2>(c, dst, src); }
int B3(atm3_ctx &c, double *dst, const double *p, double cB, int mode) {
  k3_B<<<(c.nc + CB_B - 1) / CB_B, 24 * CB_B, 0, c.stream>>>(dst, p, cB, c.ainv, mode, c.wb, c.nbt,
                                                           c.g);
  ATM_CHECK_LAUNCH("k3_B");
  return ATM_OK;
}
// after every change of pres_fix
int prep_C3(atm3_ctx &c) {
  k3_prep_C<<<(c.nc + 7) / 8, 192, 0, c.stream>>>(c.cm, c.pres_fix, c.g);
  ATM_CHECK_LAUNCH("k3_prep_C");
  return ATM_OK;
}
int CD3(atm3_ctx &c, double *dst, const double *w, const double *p, double cC, int mode) {
  std::lock_guard<std::mutex> lock(c.pair);
  k3_face_C<<<fblocks(c), NF * FPB, 0, c.stream>>>(c.fbuf, w, c.pres_fix, c.g);
  ATM_CHECK_LAUNCH("k3_face_C");
  k3_CD<<<(c.nc + CB_CD - 1) / CB_CD, 32 * CB_CD, 0, c.stream>>>(dst, w, p, cC, c.invd, mode, c.cm,
                                                               c.dm, c.fbuf, c.g);
  ATM_CHECK_LAUNCH("k3_CD");
  return ATM_OK;
}
int block_apply3(atm3_ctx &c, double *dst, const double *src, const double *inv, int ncomp,
                 double scale) {
  k3_block_apply<<<blocks(c.nc), 128, 0, c.stream>>>(dst, src, inv, ncomp, scale, c.nc);
  ATM_CHECK_LAUNCH("k3_block_apply");
  return ATM_OK;
}
int rebuild_ainv3(atm3_ctx &c) {
  k3_block_inverse<<<blocks(c.nc), 128, 0, c.stream>>>(c.ainv, c.rho_fix, c.g);
  ATM_CHECK_LAUNCH("k3_block_inverse");
  return ATM_OK;
}
// S p = D p - C A^{-1} B p (with `precondition`: times diag(D)^{-1})
int schur3(atm3_ctx &c, double *dst, const double *p, bool precondition) {
  const double co = icoef3(c);
  TRY3(B3(c, c.wv1, p, co * c.dt / (c.Ma * c.Ma), 2));
  return CD3(c, dst, c.wv1, p, co * c.dt, precondition ? 2 : 1);
}
int vmult3(atm3_ctx &c, double *dst, const double *src) {
  switch (c.nsstage) {
    case 1:
    case 4: k3_mass<<<blocks(c.nc), 128, 0, c.stream>>>(dst, src, 1, nullptr, 1.0, c.g); break;
    case 2: return schur3(c, dst, src, false);
    case 3:
    case 5: k3_mass<<<blocks(c.nc), 128, 0, c.stream>>>(dst, src, 3, c.rho_fix, 1.0, c.g); break;
    case 6:
      k3_mass<<<blocks(c.nc), 128, 0, c.stream>>>(dst, src, 1, nullptr, 1.0 / (GAS_GAMMA - 1.0), c.g);
      break;
    default: set_error("NS stage out of range"); return ATM_BAD_ARG;
  }
  ATM_CHECK_LAUNCH("k3_mass");
  return ATM_OK;
}

// GMRES(28) + left Jacobi on diag(D), CGS2 (arnoldi_step), Givens; the
// algorithm of the 2D path's gmres_schur on the 3D operator
int gmres3(atm3_ctx &c, double *x, const double *b, double tol, int maxit, int *its, double *res) {
  const long n = c.ns();
  const int m = RESTART3;
  double *V = c.krylov, *w = c.ws1, *t = c.ws2;
  double *nsq = c.dsmall + 64, *ydev = c.dsmall + 96;
  std::vector<double> H((m + 1) * m, 0.0), cs(m), sn(m), g(m + 1), y(m), hcol(m + 1);
  *its = 0;
  *res = 0.0;
  for (;;) {
    TRY3(schur3(c, t, x, false));
    TRY3(vec_xmy_scaled(c.stream, V, c.invd, b, t, n));
    TRY3(vec_dot(c.stream, V, V, n, c.red, nsq));
    TRY3(read3(c, nsq, 1));
    const double beta = std::sqrt(c.h_red[0]);
    *res = beta;
    if (!std::isfinite(beta)) { set_error("GMRES: non-finite residual"); return ATM_NONFINITE; }
    if (beta <= tol) return ATM_OK;
    if (*its >= maxit) return ATM_NOT_CONVERGED;
    TRY3(vec_scale_by_inv_norm(c.stream, V, V, nsq, n));
    std::fill(g.begin(), g.end(), 0.0);
    g[0] = beta;
    int jend = 0;
    bool done = false;
    for (int j = 0; j < m; ++j) {
      ++*its;
      TRY3(schur3(c, w, V + (long)j * n, true));
      double hn = 0.0;
      TRY3(arnoldi_step(c.stream, V, n, j, w, c.red, c.dsmall, c.h_red, hcol.data(), &hn));
      for (int l = 0; l <= j; ++l) H[l * m + j] = hcol[l];
      if (!std::isfinite(hn)) { set_error("GMRES: non-finite Arnoldi vector"); return ATM_NONFINITE; }
      H[(j + 1) * m + j] = hn;
      for (int l = 0; l < j; ++l) {
        const double a = H[l * m + j], bb = H[(l + 1) * m + j];
        H[l * m + j] = cs[l] * a + sn[l] * bb;
        H[(l + 1) * m + j] = -sn[l] * a + cs[l] * bb;
      }
      const double a = H[j * m + j], bb = H[(j + 1) * m + j];
      const double r = std::sqrt(a * a + bb * bb);
      cs[j] = a / r;
      sn[j] = bb / r;
      H[j * m + j] = r;
      H[(j + 1) * m + j] = 0.0;
      g[j + 1] = -sn[j] * g[j];
      g[j] = cs[j] * g[j];
      jend = j + 1;
      *res = std::fabs(g[j + 1]);
      if (*res <= tol || hn == 0.0 || *its >= maxit) { done = true; break; }
    }
    for (int l = jend - 1; l >= 0; --l) {
      double s = g[l];
      for (int k = l + 1; k < jend; ++k) s -= H[l * m + k] * y[k];
      y[l] = s / H[l * m + l];
    }
    ATM_CUDA(cudaMemcpyAsync(ydev, y.data(), jend * sizeof(double), cudaMemcpyHostToDevice,
                             c.stream));
    TRY3(vec_multiaxpy(c.stream, x, V, n, jend, ydev, 1.0, n));
    ATM_CUDA(cudaStreamSynchronize(c.stream));
    if (done && !c.true_check)
      return (*res <= tol) ? ATM_OK : (*its >= maxit ? ATM_NOT_CONVERGED : ATM_OK);
  }
}

// ---- the IMEX step (Atmospheric_Flow.cc:430-871, 1100-1257) ---------------
int update_density3(atm3_ctx &c) {
  if (c.hstage == 1) {
    const double *s[] = {c.rho_old, c.u_old};
    TRY3(rhs_rho3(c, c.rhs_rho, s));
    return block_apply3(c, c.rho_2, c.rhs_rho, c.minv, 1, 1.0);
  }
  if (c.hstage == 2) {
    const double *s[] = {c.rho_old, c.u_old, c.rho_2, c.u_2};
    TRY3(rhs_rho3(c, c.rhs_rho, s));
    return block_apply3(c, c.rho_3, c.rhs_rho, c.minv, 1, 1.0);
  }
  const double *s[] = {c.rho_old, c.u_old, c.rho_2, c.u_2, c.rho_3, c.u_3};
  TRY3(rhs_rho3(c, c.rhs_rho, s));
  return block_apply3(c, c.rho_cur, c.rhs_rho, c.minv, 1, 1.0);
}
int set_rho_fixed3(atm3_ctx &c, const double *rho) {
  TRY3(vec_copy(c.stream, c.rho_fix, rho, c.ns()));
  return rebuild_ainv3(c);
}
int pressure_fixed_point3(atm3_ctx &c) {
  const long ns = c.ns();
  TRY3(vec_copy(c.stream, c.pres_fix, c.p_fix_old, ns));
  TRY3(prep_C3(c));
  if (c.hstage == 1) {
    const double *sp[] = {c.rho_old, c.u_old, c.p_old, c.rho_2, c.u_fixd};
    TRY3(rhs_pres3(c, c.rhs_p, sp));
    const double *su[] = {c.rho_old, c.u_old, c.p_old, c.rho_2};
    TRY3(rhs_vel3(c, c.rhs_u, su));
  } else {
    const double *sp[] = {c.rho_old, c.u_old, c.p_old, c.rho_2, c.u_2, c.p_2, c.rho_3, c.u_fixd};
    TRY3(rhs_pres3(c, c.rhs_p, sp));
    const double *su[] = {c.rho_old, c.u_old, c.p_old, c.rho_2, c.u_2, c.p_2, c.rho_3};
    TRY3(rhs_vel3(c, c.rhs_u, su));
  }
  TRY3(block_apply3(c, c.tmp_1, c.rhs_u, c.ainv, 3, 1.0));
  const double cc = icoef3(c);
  TRY3(CD3(c, c.rhs_p, c.tmp_1, nullptr, cc * c.dt, 3));
  // SolverControl(eps |rhs|) on the Jacobi-scaled residual
  // (Atmospheric_Flow.cc:656-672); with scaled_tol, eps |diag(D)^{-1} rhs|
  double nb2;
  if (c.scaled_tol) {
    TRY3(vec_fill(c.stream, c.ws1, 0.0, ns));
    TRY3(vec_xmy_scaled(c.stream, c.ws2, c.invd, c.rhs_p, c.ws1, ns));
    TRY3(vec_dot(c.stream, c.ws2, c.ws2, ns, c.red, c.red_out));
  } else {
    TRY3(vec_dot(c.stream, c.rhs_p, c.rhs_p, ns, c.red, c.red_out));
  }
  TRY3(read3(c, c.red_out, 1));
  nb2 = c.h_red[0];
  const double tol = c.eps * std::sqrt(nb2);
  TRY3(vec_copy(c.stream, c.p_fix, c.p_fix_old, ns));
  int its = 0;
  double res = 0.0;
  int rc = gmres3(c, c.p_fix, c.rhs_p, tol, c.max_its, &its, &res);
  c.krylov_total += its;
  if (rc == ATM_NOT_CONVERGED) {
    ++c.failures;
    char msg[200];
    std::snprintf(msg, sizeof msg, "shell: Schur solve did not converge in stage %d of step %ld "
                  "(%d iterations, residual %.3e > %.3e)", c.hstage, c.steps + 1, its, res, tol);
    set_error(msg);
  }
  return rc;
}
int update_velocity3(atm3_ctx &c) {
  if (c.hstage == 1 || c.hstage == 2) {
    TRY3(B3(c, c.rhs_u, c.p_fix, icoef3(c) * c.dt / (c.Ma * c.Ma), 1));
    return block_apply3(c, c.u_fixd, c.rhs_u, c.ainv, 3, 1.0);
  }
  const double *su[] = {c.rho_old, c.u_old, c.p_old, c.rho_2, c.u_2, c.p_2, c.rho_3, c.u_3, c.p_3};
  TRY3(rhs_vel3(c, c.rhs_u, su));
  return block_apply3(c, c.u_cur, c.rhs_u, c.ainv, 3, 1.0);
}
int update_pressure3(atm3_ctx &c) {
  const double *sp[] = {c.rho_old, c.u_old, c.p_old, c.rho_2, c.u_2, c.p_2, c.rho_3, c.u_3,
                        c.p_3, c.rho_cur, c.u_cur};
  TRY3(rhs_pres3(c, c.rhs_p, sp));
  return block_apply3(c, c.p_old, c.rhs_p, c.minv, 1, GAS_GAMMA - 1.0);
}
int picard3(atm3_ctx &c) {
  const long ns = c.ns();
  for (int it = 0; it < 100; ++it) {
    TRY3(pressure_fixed_point3(c));
    TRY3(update_velocity3(c));
    ++c.picard_total;
    TRY3(vec_maxdiff(c.stream, c.p_fix, c.p_fix_old, ns, c.red, c.red_out));
    TRY3(read3(c, c.red_out, 2));
    const double err = c.h_red[0] / (c.h_red[1] + 1e-10);
    if (!std::isfinite(err)) { set_error("shell: non-finite Picard update"); return ATM_NONFINITE; }
    if (err < 1e-10) break;
    TRY3(vec_copy(c.stream, c.p_fix_old, c.p_fix, ns));
  }
  return ATM_OK;
}
int step3(atm3_ctx &c) {
  const long ns = c.ns(), nv = c.nv();
  c.hstage = 1;
  TRY3(update_density3(c));
  TRY3(set_rho_fixed3(c, c.rho_2));
  TRY3(vec_copy(c.stream, c.p_fix_old, c.p_old, ns));
  TRY3(vec_copy(c.stream, c.u_fixd, c.u_old, nv));
  TRY3(picard3(c));
  TRY3(vec_copy(c.stream, c.p_2, c.p_fix, ns));
  TRY3(vec_copy(c.stream, c.u_2, c.u_fixd, nv));
  c.hstage = 2;
  TRY3(update_density3(c));
  TRY3(set_rho_fixed3(c, c.rho_3));
  TRY3(vec_copy(c.stream, c.p_fix_old, c.p_2, ns));
  TRY3(vec_copy(c.stream, c.u_fixd, c.u_2, nv));
  TRY3(picard3(c));
  TRY3(vec_copy(c.stream, c.p_3, c.p_fix, ns));
  TRY3(vec_copy(c.stream, c.u_3, c.u_fixd, nv));
  c.hstage = 3;
  TRY3(update_density3(c));
  TRY3(set_rho_fixed3(c, c.rho_cur));
  TRY3(update_velocity3(c));
  TRY3(update_pressure3(c));
  TRY3(vec_copy(c.stream, c.rho_old, c.rho_cur, ns));
  TRY3(vec_copy(c.stream, c.u_old, c.u_cur, nv));
  ++c.steps;
  return ATM_OK;
}

}  // namespace

// ============================================================================
// C ABI (declared in include/atm_gb300.h)
// ============================================================================
extern "C" {

int atm3_ctx_create(int n_cells, const double *nodes, int n_inner, const int *inner,
                    const int *face_perm, int n_bdry, const int *bdry, atm3_ctx **out) {
  if (!out || !nodes || n_cells < 1 || (n_inner > 0 && (!inner || !face_perm)) ||
      (n_bdry > 0 && !bdry)) {
    set_error("atm3_ctx_create: bad arguments");
    return ATM_BAD_ARG;
  }
  *out = nullptr;
  // tables: every cell face listed exactly once (inner faces from both sides)
  std::vector<int> nbr(6L * n_cells, -2), nbf(6L * n_cells, -1), nperm(54L * n_cells, 0);
  auto bad = [&](const std::string &m) { set_error("atm3_ctx_create: " + m); return ATM_BAD_ARG; };
  for (int f = 0; f < n_inner; ++f) {
    const int cp = inner[4 * f], fp = inner[4 * f + 1], cm = inner[4 * f + 2], fm = inner[4 * f + 3];
    if (cp < 0 || cp >= n_cells || cm < 0 || cm >= n_cells || fp < 0 || fp > 5 || fm < 0 || fm > 5)
      return bad("inner face " + std::to_string(f) + " out of range");
    if (nbr[6 * cp + fp] != -2 || nbr[6 * cm + fm] != -2)
      return bad("cell face listed twice (inner face " + std::to_string(f) + ")");
    nbr[6 * cp + fp] = cm; nbf[6 * cp + fp] = fm;
    nbr[6 * cm + fm] = cp; nbf[6 * cm + fm] = fp;
    int seen = 0;
    for (int q = 0; q < 9; ++q) {
      const int qm = face_perm[9 * f + q];
      if (qm < 0 || qm > 8 || (seen >> qm) & 1) return bad("face_perm of face " + std::to_string(f) + " is not a permutation");
      seen |= 1 << qm;
      nperm[(6 * cp + fp) * 9 + q] = qm;
      nperm[(6 * cm + fm) * 9 + qm] = q;
    }
  }
  for (int f = 0; f < n_bdry; ++f) {
    const int c = bdry[3 * f], lf = bdry[3 * f + 1];
    if (c < 0 || c >= n_cells || lf < 0 || lf > 5) return bad("boundary face out of range");
    if (nbr[6 * c + lf] != -2) return bad("cell face listed twice (boundary)");
    nbr[6 * c + lf] = -1;
  }
  for (int i = 0; i < 6 * n_cells; ++i)
    if (nbr[i] == -2) return bad("cell " + std::to_string(i / 6) + " face " + std::to_string(i % 6) + " is not listed");
  // geometry
  const double s = std::sqrt(0.6);
  const double gx[3] = {0.5 * (1.0 - s), 0.5, 0.5 * (1.0 + s)}, gw[3] = {5.0 / 18, 8.0 / 18, 5.0 / 18};
  std::vector<double> cg((size_t)n_cells * NQ * 13), fg((size_t)n_cells * 6 * NF * 4);
  for (int c = 0; c < n_cells; ++c) {
    const double *X = nodes + 81L * c;
    for (int q = 0; q < NQ; ++q) {
      const double xi[3] = {gx[q % 3], gx[(q / 3) % 3], gx[q / 9]};
      double x[3], J[3][3], Ji[3][3];
      map3(X, xi, x, J);
      const double det = inv3(J, Ji);
      if (!(det > 0.0)) return bad("non-positive Jacobian in cell " + std::to_string(c));
      const double jw = det * gw[q % 3] * gw[(q / 3) % 3] * gw[q / 9];
      double *o = &cg[((size_t)c * NQ + q) * 13];
      for (int e = 0; e < 3; ++e)
        for (int i = 0; i < 3; ++i) o[3 * e + i] = Ji[e][i] * jw;
      o[9] = jw;
      const double r = std::sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
      for (int i = 0; i < 3; ++i) o[10 + i] = x[i] / r * EARTH_A * EARTH_A / (r * r);
    }
    for (int f = 0; f < 6; ++f)
      for (int q = 0; q < NF; ++q) {
        const int d = f / 2, t0 = d == 0 ? 1 : 0, t1 = d == 2 ? 1 : 2;
        double xi[3];
        xi[d] = (double)(f % 2);
        xi[t0] = gx[q % 3];
        xi[t1] = gx[q / 3];
        double x[3], J[3][3], Ji[3][3];
        map3(X, xi, x, J);
        const double det = inv3(J, Ji);
        double len = 0.0;
        for (int i = 0; i < 3; ++i) len += Ji[d][i] * Ji[d][i];
        len = std::sqrt(len);
        const double sg = (f % 2) ? 1.0 : -1.0;
        double *o = &fg[(((size_t)c * 6 + f) * NF + q) * 4];
        for (int i = 0; i < 3; ++i) o[i] = sg * Ji[d][i] / len;
        o[3] = det * len * gw[q % 3] * gw[q / 3];
      }
  }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    set_error("atm3_ctx_create: no CUDA device (there is no CPU path)");
    return ATM_CUDA_ERROR;
  }
  atm3_ctx *c = new atm3_ctx();
  auto fail = [&](int rc) { free3(c); return rc; };
  cudaGetDevice(&c->device);
  c->nc = n_cells;
  c->tab = Tableau::make();
  int rc = upload_tables3();
  if (rc) return fail(rc);
  if ((rc = alloc3(*c, &c->cg, cg.size())) || (rc = alloc3(*c, &c->fg, fg.size()))) return fail(rc);
  if (cudaMalloc(&c->nbr, nbr.size() * sizeof(int)) || cudaMalloc(&c->nbf, nbf.size() * sizeof(int)) ||
      cudaMalloc(&c->nperm, nperm.size() * sizeof(int)))
    return fail(cuda_fail(cudaErrorMemoryAllocation, "cudaMalloc shell tables"));
  cudaMemcpy(c->cg, cg.data(), cg.size() * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(c->fg, fg.data(), fg.size() * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(c->nbr, nbr.data(), nbr.size() * sizeof(int), cudaMemcpyHostToDevice);
  cudaMemcpy(c->nbf, nbf.data(), nbf.size() * sizeof(int), cudaMemcpyHostToDevice);
  if (cudaMemcpy(c->nperm, nperm.data(), nperm.size() * sizeof(int), cudaMemcpyHostToDevice))
    return fail(cuda_fail(cudaGetLastError(), "upload shell tables"));
  std::vector<int> own;
  for (int f = 0; f < n_inner; ++f) own.push_back(6 * inner[4 * f] + inner[4 * f + 1]);
  for (int f = 0; f < n_bdry; ++f) own.push_back(6 * bdry[3 * f] + bdry[3 * f + 1]);
  if (cudaMalloc(&c->own, own.size() * sizeof(int)) ||
      cudaMemcpy(c->own, own.data(), own.size() * sizeof(int), cudaMemcpyHostToDevice))
    return fail(cuda_fail(cudaGetLastError(), "upload shell tables"));
  c->g = Geo3{n_cells, c->cg, c->fg, c->nbr, c->nbf, c->nperm, (int)own.size(), c->own};
  const long ns = c->ns(), nv = c->nv();
  double **sv[] = {&c->rho_fix, &c->pres_fix, &c->invd, &c->ws1, &c->ws2};
  for (double **p : sv)
    if ((rc = alloc3(*c, p, ns))) return fail(rc);
  if ((rc = alloc3(*c, &c->u_fix, nv)) || (rc = alloc3(*c, &c->wv1, nv)) ||
      (rc = alloc3(*c, &c->minv, (size_t)n_cells * 64)) ||
      (rc = alloc3(*c, &c->ainv, (size_t)n_cells * 64)) ||
      (rc = alloc3(*c, &c->red, 32 * RED_BLOCKS)) || (rc = alloc3(*c, &c->red_out, 64)) ||
      (rc = alloc3(*c, &c->dsmall, 256)) || (rc = alloc3(*c, &c->wb, (size_t)n_cells * 192)) ||
      (rc = alloc3(*c, &c->nbt, (size_t)n_cells * 288)) ||
      (rc = alloc3(*c, &c->dm, (size_t)n_cells * 64)) ||
      (rc = alloc3(*c, &c->cm, (size_t)n_cells * 192)) ||
      (rc = alloc3(*c, &c->fbuf, (size_t)n_cells * 72)) ||
      (rc = alloc3(*c, &c->krylov, (size_t)(RESTART3 + 1) * ns)))
    return fail(rc);
  if (cudaMallocHost(&c->h_red, 256 * sizeof(double)) != cudaSuccess)
    return fail(cuda_fail(cudaErrorMemoryAllocation, "cudaMallocHost"));
  k3_block_inverse<<<blocks(n_cells), 128, 0, c->stream>>>(c->minv, nullptr, c->g);
  k3_invdiag_D<<<blocks(n_cells), 128, 0, c->stream>>>(c->invd, c->g);
  k3_tables<<<blocks(24 * n_cells), 128, 0, c->stream>>>(c->wb, c->nbt, c->dm, c->g);
  g_kernel_launches.fetch_add(3);
  if (cudaStreamSynchronize(c->stream) != cudaSuccess)
    return fail(cuda_fail(cudaGetLastError(), "shell set-up kernels"));
  *out = c;
  return ATM_OK;
}

int atm3_ctx_destroy(atm3_ctx *h) {
  free3(h);
  return ATM_OK;
}

int atm3_set_params(atm3_ctx *h, double dt, double mach, double froude) {
  if (!h || !(dt > 0) || !(mach > 0) || !(froude > 0)) {
    set_error("atm3_set_params: null handle or non-positive value");
    return ATM_BAD_ARG;
  }
  h->dt = dt; h->Ma = mach; h->Fr = froude;
  return ATM_OK;
}

int atm3_set_stage(atm3_ctx *h, int hyperbolic_stage, int ns_stage) {
  if (!h || hyperbolic_stage < 1 || hyperbolic_stage > 3 || ns_stage < 1 || ns_stage > 6) {
    set_error("atm3_set_stage: null handle or stage out of range");
    return ATM_BAD_ARG;
  }
  h->hstage = hyperbolic_stage;
  h->nsstage = ns_stage;
  return ATM_OK;
}

int atm3_set_frozen(atm3_ctx *h, const double *rho, const double *pres, const double *u) {
  if (!h) { set_error("null handle"); return ATM_BAD_ARG; }
  if (rho) {
    ATM_CUDA(cudaMemcpyAsync(h->rho_fix, rho, h->ns() * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
    int rc = rebuild_ainv3(*h);
    if (rc) return rc;
  }
  if (pres) {
    ATM_CUDA(cudaMemcpyAsync(h->pres_fix, pres, h->ns() * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
    if (int rc = prep_C3(*h)) return rc;
  }
  if (u) ATM_CUDA(cudaMemcpyAsync(h->u_fix, u, h->nv() * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  return ATM_OK;
}

int atm3_rhs(atm3_ctx *h, int which, double *dst, const double *const *src, int nsrc) {
  if (!h || !dst || !src || which < 0 || which > 2) {
    set_error("atm3_rhs: bad arguments");
    return ATM_BAD_ARG;
  }
  static const int need[3][3] = {{2, 4, 6}, {4, 7, 9}, {5, 8, 11}};
  if (nsrc != need[which][h->hstage - 1]) {
    set_error("atm3_rhs: wrong number of sources for this equation and IMEX stage");
    return ATM_BAD_ARG;
  }
  for (int i = 0; i < nsrc; ++i)
    if (!src[i]) { set_error("atm3_rhs: null source"); return ATM_BAD_ARG; }
  int rc = which == 0 ? rhs_rho3(*h, dst, src) : which == 1 ? rhs_vel3(*h, dst, src)
                                                          : rhs_pres3(*h, dst, src);
  if (rc) return rc;
  ATM_CUDA(cudaStreamSynchronize(h->stream));
  return ATM_OK;
}

int atm3_apply(atm3_ctx *h, int which, double *dst, const double *src) {
  if (!h || !dst || !src || which < 0 || which > 2) {
    set_error("atm3_apply: bad arguments");
    return ATM_BAD_ARG;
  }
  int rc;
  if (which == 0) rc = B3(*h, dst, src, icoef3(*h) * h->dt / (h->Ma * h->Ma), 0);
  else if (which == 1) rc = CD3(*h, dst, src, nullptr, icoef3(*h) * h->dt, 0);
  else rc = vmult3(*h, dst, src);
  if (rc) return rc;
  ATM_CUDA(cudaStreamSynchronize(h->stream));
  return ATM_OK;
}

int atm3_solver_init(atm3_ctx *h, double eps, int max_its, int scaled_tol, int true_residual_check) {
  if (!h || !(eps > 0.0) || max_its < 1) {
    set_error("atm3_solver_init: null handle, eps <= 0 or max_its < 1");
    return ATM_BAD_ARG;
  }
  if (!h->pool) {
    const long ns = h->ns(), nv = h->nv();
    int rc = alloc3(*h, &h->pool, 11 * ns + 7 * nv);
    if (rc) return rc;
    double *p = h->pool;
    auto take = [&](long n) { double *r = p; p += n; return r; };
    h->rho_old = take(ns); h->rho_2 = take(ns); h->rho_3 = take(ns); h->rho_cur = take(ns);
    h->rhs_rho = take(ns); h->p_old = take(ns); h->p_2 = take(ns); h->p_3 = take(ns);
    h->p_fix = take(ns); h->p_fix_old = take(ns); h->rhs_p = take(ns);
    h->u_old = take(nv); h->u_2 = take(nv); h->u_3 = take(nv); h->u_cur = take(nv);
    h->u_fixd = take(nv); h->rhs_u = take(nv); h->tmp_1 = take(nv);
  }
  h->solver = true;
  h->eps = eps;
  h->max_its = max_its;
  h->scaled_tol = scaled_tol != 0;
  h->true_check = true_residual_check != 0;
  h->steps = h->picard_total = h->krylov_total = h->failures = 0;
  return ATM_OK;
}

int atm3_solver_set_state(atm3_ctx *h, const double *rho, const double *u, const double *p) {
  if (!h || !h->solver || !rho || !u || !p) {
    set_error("atm3_solver_set_state: solver not initialised or null pointer");
    return ATM_BAD_ARG;
  }
  ATM_CUDA(cudaMemcpy(h->rho_old, rho, h->ns() * sizeof(double), cudaMemcpyHostToDevice));
  ATM_CUDA(cudaMemcpy(h->u_old, u, h->nv() * sizeof(double), cudaMemcpyHostToDevice));
  ATM_CUDA(cudaMemcpy(h->p_old, p, h->ns() * sizeof(double), cudaMemcpyHostToDevice));
  return ATM_OK;
}

int atm3_solver_get_state(atm3_ctx *h, double *rho, double *u, double *p) {
  if (!h || !h->solver || !rho || !u || !p) {
    set_error("atm3_solver_get_state: solver not initialised or null pointer");
    return ATM_BAD_ARG;
  }
  ATM_CUDA(cudaStreamSynchronize(h->stream));
  ATM_CUDA(cudaMemcpy(rho, h->rho_old, h->ns() * sizeof(double), cudaMemcpyDeviceToHost));
  ATM_CUDA(cudaMemcpy(u, h->u_old, h->nv() * sizeof(double), cudaMemcpyDeviceToHost));
  ATM_CUDA(cudaMemcpy(p, h->p_old, h->ns() * sizeof(double), cudaMemcpyDeviceToHost));
  return ATM_OK;
}

int atm3_solver_run(atm3_ctx *h, int n_steps) {
  if (!h || !h->solver || n_steps < 0) {
    set_error("atm3_solver_run: solver not initialised or n_steps < 0");
    return ATM_BAD_ARG;
  }
  for (int i = 0; i < n_steps; ++i) {
    int rc = step3(*h);
    if (rc) return rc;
  }
  ATM_CUDA(cudaStreamSynchronize(h->stream));
  return ATM_OK;
}

int atm3_solver_stats(atm3_ctx *h, double *out) {
  if (!h || !out) { set_error("null handle or pointer"); return ATM_BAD_ARG; }
  out[0] = (double)h->steps;
  out[1] = (double)h->picard_total;
  out[2] = (double)h->krylov_total;
  out[3] = (double)h->failures;
  return ATM_OK;
}

}  // extern "C"
