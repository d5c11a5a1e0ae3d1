// Schur-complement kernels for mappings of degree <= 2 (MappingQ(2),
// equation_data.h:43): B (then optionally the exact cell-wise A^{-1}) and C/D.
//   B   euler_operator.h:1512-1617
//   C   euler_operator.h:1413-1507
//   D   euler_operator.h:1386-1408
//
// The FP64 pipe of sm_103a issues two lanes per clock and SM, so a kernel
// here costs what its FP64 instructions cost; everything else hides behind
// them.  Two things set that count.
//   * Quadrature.  The reference integrates everything with QGauss(2k+1).  On
//     a degree-2 mapping the cofactors of the Jacobian have degree <= 2 along
//     their own reference direction and <= 1 along the other one, so the
//     integrands of B (p cof grad v) have degree 2k+1 and those of C
//     (w p_fix cof grad q) degree 3k+1 in each direction: k+1 and
//     NC = floor((3k+3)/2) Gauss points integrate them exactly, as the 2k+1
//     points do (D, degree 2k+3, is exact on the NC points too).  The results
//     agree to rounding with 25 and 49 points instead of 81 at k = 4.  The face
//     terms of C hold the upwind speed max |w.n|, which is no polynomial: they
//     keep the 2k+1 points.  The face terms of B (degree 2k+1) take k+1.
//   * Idle lanes cost as much as busy ones.  Every 1D contraction is done for
//     a whole row, column or face by one thread, with the even-odd split of
//     the symmetric point sets and compile-time coefficients, and the tasks of
//     a phase are dealt out over the threads of the block so that warps are
//     full: (cell, row), (cell, column), (cell, face), (cell, row of A^{-1}).
//
// Geometry enters as products tabulated once per mesh (k_exact_tables): the
// cofactors times the quadrature weight per point, four values together, and
// the outward normal times the face weight, each with the equation's constant
// factors.  p_fix enters C as H = gamma/(gamma-1) p_fix cof per point and as
// its face traces, prepared when p_fix is set.
//
// Measured on GB300 at 51,200 cells, k = 4 (before: the kernels of
// schur_kernels.cuh, 2k+1 points everywhere, 9 threads per cell): FP64 B with
// A^{-1} 0.56 -> 0.24 ms, C/D 0.55 -> 0.28 ms (63 us of it the faces), the FP64
// pipe busy 80-89%; the FP32 V-cycle 1.54 -> 0.80 ms.
//
// In the Schur apply, B stores w = cB cC A^{-1} B p and C/D applies C with unit
// coefficient: C is homogeneous of degree one in w for the positive cC
// (the upwind speed scales with w).
#pragma once
#include "contract.cuh"

namespace atm {

// flux of C at a face point, times the face weight: half gamma/(gamma-1)
// (a un+ + b un-) plus the upwind jump max |un| (a - b) / (2 (gamma-1)), with
// a, b the p_fix traces and g the normal times the weight times half
// gamma/(gamma-1)
template <typename T>
__device__ __forceinline__ T flux_C(const T *__restrict__ g, T wx, T wz, T vx, T vz, T a, T b) {
  T n0, n1;
  load2(g, n0, n1);
  const T up = fma(wx, n0, wz * n1), um = fma(vx, n0, vz * n1);
  return fma(abs_max(up, um), (a - b) * T(1.0 / GAS_GAMMA), fma(a, up, b * um));
}

// asynchronous copy of n contiguous values into shared memory by the block;
// both addresses 16-byte aligned (blocks start at multiples of 8 cells)
__device__ __forceinline__ void stage(float *s, const float *g, int n) {
  for (int e = threadIdx.x; e < n / 4; e += blockDim.x) cp_async16(s + 4 * e, g + 4 * e);
  for (int e = n / 4 * 4 + threadIdx.x; e < n; e += blockDim.x) cp_async4(s + e, g + e);
}

// face contributions of the output row iz: faces x = 0, 1 add to the row's
// ends, faces z = 0, 1 to the whole first and last row.  F: [4][NN]
template <int K, typename T>
__device__ __forceinline__ void face_rows(const T *__restrict__ F, int iz, T (&add)[K + 1]) {
  constexpr int NN = K + 1;
  const T *Fz = iz == 0 ? F + 2 * NN : F + 3 * NN;
  const bool edge = iz == 0 || iz == K;
#pragma unroll
  for (int i = 0; i < NN; ++i) add[i] = edge ? Fz[i] : T(0);
  add[0] += F[iz];
  add[K] += F[NN + iz];
}

// (rows NN of A^{-1}) x (b0, b1) of one cell, FP32 tiles: thread (cell, a) owns
// the node row iz = a, s0/s1[r] for the nodes (a, r).  b holds (b0, b1) pairs.
template <int K>
__device__ __forceinline__ void atile_apply(const float *__restrict__ A,
                                            const float2 *__restrict__ b, int a,
                                            float (&s0)[K + 1], float (&s1)[K + 1]) {
  using L = ATile<K>;
  constexpr int NN = K + 1;
#pragma unroll
  for (int r = 0; r < NN; ++r) s0[r] = s1[r] = 0.0f;
#pragma unroll
  for (int t = 0; t < NN; ++t) {
    float2 v[NN];
#pragma unroll
    for (int j = 0; j < NN; ++j) v[j] = b[t * NN + j];
    if (t == a) {
      float d[L::DIA];
#pragma unroll
      for (int i = 0; i < L::DIA; i += 4)
        *reinterpret_cast<float4 *>(d + i) =
            *reinterpret_cast<const float4 *>(A + L::D0 + t * L::DIA + i);
#pragma unroll
      for (int r = 0; r < NN; ++r)
#pragma unroll
        for (int j = 0; j < NN; ++j) {
          const float x = d[r >= j ? r * (r + 1) / 2 + j : j * (j + 1) / 2 + r];
          s0[r] = fmaf(x, v[j].x, s0[r]);
          s1[r] = fmaf(x, v[j].y, s1[r]);
        }
    } else {
      const int hi = max(a, t), lo = min(a, t);
      const float *T = A + (hi * (hi - 1) / 2 + lo) * L::OFF;
      float d[L::OFF];
#pragma unroll
      for (int i = 0; i < L::OFF; i += 4)
        *reinterpret_cast<float4 *>(d + i) = *reinterpret_cast<const float4 *>(T + i);
      if (a > t) {
#pragma unroll
        for (int r = 0; r < NN; ++r)
#pragma unroll
          for (int j = 0; j < NN; ++j) {
            s0[r] = fmaf(d[r * NN + j], v[j].x, s0[r]);
            s1[r] = fmaf(d[r * NN + j], v[j].y, s1[r]);
          }
      } else {  // the transposed tile
#pragma unroll
        for (int r = 0; r < NN; ++r)
#pragma unroll
          for (int j = 0; j < NN; ++j) {
            s0[r] = fmaf(d[j * NN + r], v[j].x, s0[r]);
            s1[r] = fmaf(d[j * NN + r], v[j].y, s1[r]);
          }
      }
    }
  }
}

// ====================================================================== B ===
// MODE 0: dst = cB B p ; 1: dst -= cB B p ; 2: dst = cB cC A^{-1} B p
// (with a per-cell time-step multiplier d: cB d and cC d).
//
// B is evaluated in its strong form: with exact quadrature
//   -int p d(phi) + oint p* n phi = int d(p) phi - oint (p - p*) n phi,
// which takes one derivative of p (six percent fewer FP64 instructions than
// testing with the gradients of both components) and has no wall term (p* = p
// there).  p - p* is half the jump of p.
//
// The first 4 cpb threads take the faces, the next (k+1) cpb the rows, then
// the columns and the output rows; A^{-1} is dealt out over all of them.
// `cpb` cells per block, a multiple of 8 (whole warps of face threads).
template <int K>
struct ExB {
  static constexpr int TPC = K + 5;         // threads per cell
  static constexpr int XV = 2 * (K + 1) * (K + 1), FV = 8 * (K + 1);
  template <typename T>
  static constexpr int values(bool stage) {  // shared-memory values per cell
    return 2 * XV + FV + (stage ? ainv_stride<K, T>() : 0);
  }
};

// nodal integrals of the face term of B over face f of cell cf, both
// components: F[0..k] and F[4(k+1)..]; without HG the face is conforming or a wall
template <int K, typename T, bool HG>
__device__ __forceinline__ void face_B(const T *__restrict__ p, const MeshT<T> &mesh, int cf,
                                       int f, T *__restrict__ F) {
  constexpr int NN = K + 1, NN2 = NN * NN;
  // fB, hB hold half the outward normal times the weight; what is added to
  // the rows is half the jump times it
  const int nb = mesh.nbr[cf * 4 + f], nfc = mesh.nbrf[cf * 4 + f];
  const int code = HG && nb >= 0 ? nfc >> 2 : 0;
  T own[NN], o0[NN], o1[NN];
#pragma unroll
  for (int i = 0; i < NN; ++i) o0[i] = o1[i] = T(0);
  if (nb >= 0) {
    trace<K, !HG>(p + (long)cf * NN2, f, own);
    if (!HG || code < 3) {
      T nbt[NN], s[NN], F0[NN], F1[NN];
      trace<K, !HG>(p + (long)nb * NN2, nfc & 3, nbt);
      if (!HG || code == 0) {
#pragma unroll
        for (int i = 0; i < NN; ++i) nbt[i] -= own[i];
        eo_interp<K, 0>(nbt, s);
      } else {  // fine side: the coarse neighbour at the shifted points
        T sn[NN];
        eo_interp<K, 0>(own, sn);
        sub_interp<K, 0>(nbt, code - 1, s);
#pragma unroll
        for (int q = 0; q < NN; ++q) s[q] -= sn[q];
      }
      const T *g = mesh.fB + ((long)cf * 4 + f) * 2 * NN;
#pragma unroll
      for (int q = 0; q < NN; ++q) {
        T n0, n1;
        load2(g + 2 * q, n0, n1);
        F0[q] = n0 * s[q];
        F1[q] = n1 * s[q];
      }
      eo_integ<K, 0, NN, true, false>(F0, F0, o0);
      eo_integ<K, 0, NN, true, false>(F1, F1, o1);
    } else {  // coarse side: two subfaces
      for (int h = 0; h < 2; ++h) {
        T nbt[NN], s[NN], sn[NN], F0[NN], F1[NN];
        trace<K>(p + (long)mesh.hnb[nb * 2 + h] * NN2, nfc & 3, nbt);
        sub_interp<K, 0>(own, h, sn);
        eo_interp<K, 0>(nbt, s);
        const T *g = mesh.hB + ((long)nb * 2 + h) * 2 * NN;
#pragma unroll
        for (int q = 0; q < NN; ++q) {
          T n0, n1;
          load2(g + 2 * q, n0, n1);
          s[q] -= sn[q];
          F0[q] = n0 * s[q];
          F1[q] = n1 * s[q];
        }
        sub_integ_add<K, 0>(F0, h, o0);
        sub_integ_add<K, 0>(F1, h, o1);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NN; ++i) {
    F[i] = o0[i];
    F[4 * NN + i] = o1[i];
  }
}

template <int K, int MODE, typename T, bool HG>
__global__ void __launch_bounds__(320)
    k_exact_B(T *__restrict__ dst, const T *__restrict__ p, T cB, T cC,
              const T *__restrict__ ainv, MeshT<T> mesh, int cpb) {
  constexpr int NN = K + 1, NN2 = NN * NN, XV = ExB<K>::XV, FV = ExB<K>::FV;
  constexpr bool STAGE = MODE == 2 && sizeof(T) == 4;
  constexpr int AS = ainv_stride<K, T>();
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T *sm = reinterpret_cast<T *>(sm_raw);
  T *as = sm;                                // [cpb][AS] staged A^{-1} (STAGE)
  T *Xs = sm + (STAGE ? cpb * AS : 0);       // [cpb][2][NN2] p, d_xi p at (iz, qx); then B p pairs
  T *Y = Xs + cpb * XV;                      // [cpb][2 comp][NN2]; then the result
  T *Fs = Y + cpb * XV;                      // [cpb][2 comp][4][NN]
  int *hlist = reinterpret_cast<int *>(Fs + cpb * FV);  // count, hanging faces (HG)
  const int tid = threadIdx.x;
  const int c0 = blockIdx.x * cpb;
  const int cnt = min(cpb, mesh.nc - c0);
  pdl_trigger();  // C/D may take the slots that the tail of this grid leaves
  if constexpr (STAGE) {
    // cells c0 .. c0+cnt-1: cnt * AS values, 16-byte aligned (AS % 4 == 0);
    // they arrive while B is computed
    const T *src = ainv + (long)c0 * AS;
    const int n16 = cnt * AS / 4;
    for (int e = tid; e < n16; e += blockDim.x) cp_async16(as + 4 * e, src + 4 * e);
    cp_async_commit();
  }
  // up to here only A^{-1} (FP32): on a level at least one kernel launched without
  // overlap (k_mg_start, k_restrict, k_hash_init) lies between k_block_inverse and
  // every B
  pdl_wait();
  if constexpr (HG) {
    if (tid == 0) hlist[0] = 0;
    __syncthreads();
  }
  const int rt = tid - 4 * cpb;             // row/column threads: rt >= 0
  const int lc = rt / NN, j = rt - lc * NN;
  const bool active = rt >= 0 && lc < cnt;
  const int c = c0 + lc;
  if (active) {
    // row j: values and xi-derivatives at the k+1 Gauss points
    T t[NN], v[NN], d[NN];
    const T *row = p + (long)c * NN2 + j * NN;
#pragma unroll
    for (int i = 0; i < NN; ++i) t[i] = load_late(row + i);
    eo_interp_d<K, 0>(t, v, d);
    T *x = Xs + lc * XV + j * NN;
#pragma unroll
    for (int i = 0; i < NN; ++i) {
      x[i] = v[i];
      x[NN2 + i] = d[i];
    }
  } else if (rt < 0 && tid < 4 * cnt) {
    const int l = tid >> 2, f = tid & 3;
    if (HG && mesh.nbr[(c0 + l) * 4 + f] >= 0 && (mesh.nbrf[(c0 + l) * 4 + f] >> 2) != 0)
      hlist[1 + atomicAdd(hlist, 1)] = tid;
    else
      face_B<K, T, false>(p, mesh, c0 + l, f, Fs + l * FV + f * NN);
  }
  __syncthreads();
  if constexpr (HG)
    for (int t = tid; t < hlist[0]; t += blockDim.x) {
      const int l = hlist[1 + t] >> 2, f = hlist[1 + t] & 3;
      face_B<K, T, true>(p, mesh, c0 + l, f, Fs + l * FV + f * NN);
    }
  if (active) {
    // column j: gradient at the points, z-integration of both components
    T t[NN], px[NN], pe[NN], G0[NN], G1[NN], b[NN];
    const T *x = Xs + lc * XV + j;
#pragma unroll
    for (int i = 0; i < NN; ++i) t[i] = x[NN2 + i * NN];
    eo_interp<K, 0>(t, px);
#pragma unroll
    for (int i = 0; i < NN; ++i) t[i] = x[i * NN];
    eo_deriv<K, 0>(t, pe);
    const T *g = mesh.gB + ((long)c * NN + j) * NN * 4;
#pragma unroll
    for (int q = 0; q < NN; ++q) {
      const Vec4<T> w(g + 4 * q);  // cofactors of (xi, eta) for d/dx, then for d/dz
      G0[q] = fma(w.v[0], px[q], w.v[1] * pe[q]);
      G1[q] = fma(w.v[2], px[q], w.v[3] * pe[q]);
    }
    T *y = Y + lc * XV + j;
    eo_integ<K, 0, NN, true, false>(G0, G0, b);
#pragma unroll
    for (int i = 0; i < NN; ++i) y[i * NN] = b[i];
    eo_integ<K, 0, NN, true, false>(G1, G1, b);
#pragma unroll
    for (int i = 0; i < NN; ++i) y[NN2 + i * NN] = b[i];
  }
  __syncthreads();
  if (active) {
    // output row j; MODE 2 leaves (B p)_x, (B p)_z pairs in Xs
    T s = MODE == 2 ? cB * cC : cB;
    if (mesh.dts) {
      const T d = mesh.dts[c];
      s *= MODE == 2 ? d * d : d;
    }
#pragma unroll
    for (int comp = 0; comp < 2; ++comp) {
      const T *y = Y + lc * XV + comp * NN2 + j * NN;
      T a[NN], out[NN], add[NN];
#pragma unroll
      for (int i = 0; i < NN; ++i) a[i] = y[i];
      eo_integ<K, 0, NN, true, false>(a, a, out);
      face_rows<K>(Fs + lc * FV + comp * 4 * NN, j, add);
      T *d = dst + ((long)c * 2 + comp) * NN2 + j * NN;
#pragma unroll
      for (int i = 0; i < NN; ++i) {
        const T o = s * (out[i] + add[i]);
        if (MODE == 2) Xs[lc * XV + 2 * (j * NN + i) + comp] = o;
        else if (MODE == 1) d[i] -= o;
        else d[i] = o;
      }
    }
  }
  if constexpr (MODE == 2) {
    if constexpr (STAGE) cp_async_wait_all();
    __syncthreads();
    if constexpr (STAGE) {
      // thread (a, cell): the node row a of the cell, then one coalesced copy
      for (int e = tid; e < NN * cpb; e += blockDim.x) {
        const int a = e / cpb, l = e - a * cpb;
        if (l >= cnt) continue;
        T s0[NN], s1[NN];
        atile_apply<K>(as + l * AS, reinterpret_cast<const float2 *>(Xs + l * XV), a, s0, s1);
        T *y = Y + l * XV + a * NN;
#pragma unroll
        for (int r = 0; r < NN; ++r) {
          y[r] = s0[r];
          y[NN2 + r] = s1[r];
        }
      }
      __syncthreads();
      T *d = dst + (long)c0 * XV;
      for (int e = tid; e < cnt * XV; e += blockDim.x) d[e] = Y[e];
    } else {
      // rows (cell, i) of A^{-1}: consecutive threads read consecutive values
      // of the cell's (symmetric) block
      for (int e = tid; e < cnt * NN2; e += blockDim.x) {
        const int l = e / NN2, i = e - l * NN2;
        const T *b = Xs + l * XV;
        T s0 = T(0), s1 = T(0);
        const T *Ab = ainv + (long)(c0 + l) * AS + i;
#pragma unroll
        for (int jj = 0; jj < NN2; ++jj) {
          const T a = load_late(Ab + jj * NN2);
          s0 = fma(a, b[2 * jj], s0);
          s1 = fma(a, b[2 * jj + 1], s1);
        }
        T *d = dst + (long)(c0 + l) * 2 * NN2 + i;
        d[0] = s0;
        d[NN2] = s1;
      }
    }
  }
}

// nodal integrals o of C w over face f of cell c
template <int K, typename T, bool HG>
__device__ __forceinline__ void face_C(const T *__restrict__ w, const T *__restrict__ pfix,
                                       const T *__restrict__ pff, const MeshT<T> &mesh, int c,
                                       int f, T (&o)[K + 1]) {
  constexpr int NN = K + 1, NN2 = NN * NN, NQ = 2 * K + 1;
  const int nb = mesh.nbr[c * 4 + f], nfc = mesh.nbrf[c * 4 + f];
  const int code = HG && nb >= 0 ? nfc >> 2 : 0;
  const T *wc = w + (long)c * 2 * NN2;
  if (nb < 0) {
#pragma unroll
    for (int i = 0; i < NN; ++i) o[i] = T(0);
  } else if (!HG || code == 0) {
    T t[NN], wx[NQ], wz[NQ], vx[NQ], vz[NQ], F[NQ];
    const T *wn = w + (long)nb * 2 * NN2;
    trace<K, !HG>(wc, f, t);
    eo_interp<K, 2>(t, wx);
    trace<K, !HG>(wc + NN2, f, t);
    eo_interp<K, 2>(t, wz);
    trace<K, !HG>(wn, nfc & 3, t);
    eo_interp<K, 2>(t, vx);
    trace<K, !HG>(wn + NN2, nfc & 3, t);
    eo_interp<K, 2>(t, vz);
    const T *hp = pff + ((long)c * 4 + f) * NQ, *hm = pff + ((long)nb * 4 + (nfc & 3)) * NQ;
    const T *g = mesh.fC + ((long)c * 4 + f) * 2 * NQ;
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      F[q] = flux_C(g + 2 * q, wx[q], wz[q], vx[q], vz[q], load_late(hp + q), load_late(hm + q));
    eo_integ<K, 2, NQ, true, false>(F, F, o);
  } else {
#pragma unroll
    for (int i = 0; i < NN; ++i) o[i] = T(0);
    // fine side (code 1, 2): one face, the neighbour at the shifted points;
    // coarse side (code 3): two subfaces, this cell at the shifted points
    for (int h = 0; h < (code == 3 ? 2 : 1); ++h) {
      const int nc = code == 3 ? mesh.hnb[nb * 2 + h] : nb;
      const T *wn = w + (long)nc * 2 * NN2;
      T wx[NQ], wz[NQ], vx[NQ], vz[NQ], a[NQ], b[NQ], F[NQ];
      own_or_sub<K>(wc, f, code == 3 ? h : -1, wx);
      own_or_sub<K>(wc + NN2, f, code == 3 ? h : -1, wz);
      own_or_sub<K>(pfix + (long)c * NN2, f, code == 3 ? h : -1, a);
      own_or_sub<K>(wn, nfc & 3, code == 3 ? -1 : code - 1, vx);
      own_or_sub<K>(wn + NN2, nfc & 3, code == 3 ? -1 : code - 1, vz);
      own_or_sub<K>(pfix + (long)nc * NN2, nfc & 3, code == 3 ? -1 : code - 1, b);
      const T *g = code == 3 ? mesh.hC + ((long)nb * 2 + h) * 2 * NQ
                             : mesh.fC + ((long)c * 4 + f) * 2 * NQ;
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        F[q] = flux_C(g + 2 * q, wx[q], wz[q], vx[q], vz[q], a[q], b[q]);
      if (code == 3) {
        sub_integ_add<K, 1>(F, h, o);
      } else {
        eo_integ<K, 2, NQ, true, false>(F, F, o);
      }
    }
  }
}

// what face_rows adds, from the face integrals of k_exact_face_C (Fb[c][f][NN]):
// even conforming faces take the neighbour's with the sign flipped
template <int K>
__device__ __forceinline__ void face_rows_of(const double *__restrict__ Fb, const Mesh &mesh,
                                             long c, int iz, double (&add)[K + 1]) {
  constexpr int NN = K + 1;
  const int4 nb4 = *reinterpret_cast<const int4 *>(mesh.nbr + c * 4);
  const int4 nf4 = *reinterpret_cast<const int4 *>(mesh.nbrf + c * 4);
  const int nb[4] = {nb4.x, nb4.y, nb4.z, nb4.w}, nf[4] = {nf4.x, nf4.y, nf4.z, nf4.w};
#pragma unroll
  for (int i = 0; i < NN; ++i) add[i] = 0.0;
  // faces z = 0, 1 reach a row only at the first and last row
  const int fz = iz == 0 ? 2 : 3;
  const bool edge = iz == 0 || iz == K;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int f = k < 2 ? k : fz;
    const int b = k == 0 ? nb[0] : k == 1 ? nb[1] : fz == 2 ? nb[2] : nb[3];
    const int n = k == 0 ? nf[0] : k == 1 ? nf[1] : fz == 2 ? nf[2] : nf[3];
    if (b < 0 || (k == 2 && !edge)) continue;
    const bool theirs = !(f & 1) && (n >> 2) == 0;
    const double *F = Fb + (theirs ? (long)b * 4 + (n & 3) : c * 4 + f) * NN;
    const long long flip = theirs ? (long long)0x8000000000000000ull : 0;
    if (k < 2) {
      const double v = __longlong_as_double(__double_as_longlong(F[iz]) ^ flip);
      if (k == 0) add[0] = v;
      else add[K] = v;
    } else {
#pragma unroll
      for (int i = 0; i < NN; ++i)
        add[i] += __longlong_as_double(__double_as_longlong(F[i]) ^ flip);
    }
  }
}
template <int K>
__device__ __forceinline__ void face_rows_of(const float *, const MeshT<float> &, long, int,
                                             float (&)[K + 1]) {}

// ===================================================================== CD ===
// MODE 0: dst = cC C w ; 3: dst -= cC C w
// MODE 1: dst = D p - C w ; 2: dst = invd .* (D p - C w)
// MODE 4: t = D p - C w with p = ch.x, then the Chebyshev update of ch
//
// Large FP64 meshes (FB): a face takes 256 FP64 instructions at k = 4, the rest
// of a cell 2150, so k_exact_face_C integrates every conforming face once and
// this kernel reads the integrals; without its own faces it fills blocks of
// whole warps.  Smaller meshes (EXACT_FB_UNKNOWNS), calls that may not use the
// handle's workspace (C alone, the static-scratch S) and the FP32 levels (not bound
// by arithmetic) integrate their own four faces.
//
// Threads (cell, column), column < NC; `cpb` cells per block, without FB a
// multiple of 8, at most 32.  Three blocks per SM in FP64 (80 registers, k = 4):
// two leave the SM's quarters with 4, 4, 3 and 3 warps (51,200 cells: S apply 577 -> 572 us); five in FP32.
// Measured at k = 4 and applied to every order: at k = 5 the FP32 form has 40
// registers and spills 224 bytes, with a V-cycle of 0.55 ms at 160x80 (0.92 by the
// general kernels).
template <int K, int MODE, typename T, bool HG, bool FB>
__global__ void __launch_bounds__(FB ? 256 : 32 * Ex<K>::NC, FB ? 3 : HG ? 1 : sizeof(T) == 8 ? 3 : 5)
    k_exact_CD(T *__restrict__ dst, const T *__restrict__ w, const T *__restrict__ p,
               const T *__restrict__ pfix, const T *__restrict__ hq, const T *__restrict__ pff,
               const T *__restrict__ Fb, T cC, const T *__restrict__ invd, MeshT<T> mesh,
               ChebArgs<T> ch, int cpb) {
  using E = Ex<K>;
  constexpr int NN = E::NN, NN2 = E::NN2, NC = E::NC, NC2 = E::NC2, NQ = E::NQ;
  constexpr bool WITH_D = MODE == 1 || MODE == 2 || MODE == 4;
  constexpr int NF = WITH_D ? 3 : 2;
  constexpr int XS = NN * NC;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  // FP32 (multigrid levels, latency bound): H, det J and the Chebyshev vectors
  // of the block's cells are contiguous and arrive in shared memory while the
  // faces and rows are computed (V-cycle of 320x160, k = 4: 0.90 -> 0.84 ms)
  constexpr bool STG = sizeof(T) == 4;
  constexpr int NV = MODE == 4 ? 4 : 0;
  T *sH = reinterpret_cast<T *>(sm_raw);       // [cpb][NC][NC][4] (STG)
  T *sJ = sH + (STG ? cpb * 4 * NC2 : 0);      // [cpb][NC][NC]
  T *sV = sJ + (STG ? cpb * NC2 : 0);          // [NV][cpb][NN2]: rhs, invd, d, x
  T *X = sV + (STG ? NV * cpb * NN2 : 0);      // [cpb][NF][NN][NC] x-interpolated w, p; then xa, xb
  T *Fs = X + cpb * NF * XS;                   // [cpb][4][NN] face integrals of C w (not FB)
  int *hlist = reinterpret_cast<int *>(Fs + cpb * 4 * NN);  // count, hanging faces (HG)
  const int tid = threadIdx.x, nt = blockDim.x;
  const int c0 = blockIdx.x * cpb;
  const int cnt = min(cpb, mesh.nc - c0);
  if constexpr (STG) {
    // H and det J: as A^{-1} in k_exact_B, a kernel launched without overlap lies
    // between k_exact_pfix and every C/D of a level
    stage(sH, hq + (long)c0 * 4 * NC2, cnt * 4 * NC2);
    if (WITH_D) stage(sJ, mesh.gJ + (long)c0 * NC2, cnt * NC2);
  }
  pdl_wait();
  if constexpr (STG) {
    if constexpr (NV > 0) {
      stage(sV, ch.rhs + (long)c0 * NN2, cnt * NN2);
      stage(sV + cpb * NN2, invd + (long)c0 * NN2, cnt * NN2);
      stage(sV + 2 * cpb * NN2, ch.d + (long)c0 * NN2, cnt * NN2);
      stage(sV + 3 * cpb * NN2, p + (long)c0 * NN2, cnt * NN2);
    }
    cp_async_commit();
  }
  if constexpr (HG && !FB) {
    if (tid == 0) hlist[0] = 0;
    __syncthreads();
  }
  // faces: one thread per (cell, face); with NC > 4 the first 4 cpb threads
  // (whole warps) take them while the others interpolate the rows.  Hanging
  // faces take several times as long: they are put on a list and done by
  // consecutive threads, instead of holding up a warp each (S apply of 6300
  // cells with 184 hanging subfaces, k = 3: 84 -> 74 us)
  for (int e = tid; !FB && e < 4 * cnt; e += nt) {
    const int f = e & 3, c = c0 + (e >> 2);
    if (HG && mesh.nbr[c * 4 + f] >= 0 && (mesh.nbrf[c * 4 + f] >> 2) != 0) {
      hlist[1 + atomicAdd(hlist, 1)] = e;
      continue;
    }
    T o[NN];
    face_C<K, T, false>(w, pfix, pff, mesh, c, f, o);
#pragma unroll
    for (int i = 0; i < NN; ++i) Fs[e * NN + i] = o[i];
  }
  // rows (cell, field, iz): x-interpolation to the NC points
  {
    constexpr bool SPLIT = NC > 4 && !FB;
    const int first = SPLIT ? 4 * cpb : 0, stride = nt - first;
    for (int e = tid - first; e >= 0 && e < cnt * NF * NN; e += stride) {
      const int l = e / (NF * NN), r = e - l * (NF * NN);
      const T *row = r < 2 * NN ? w + ((long)(c0 + l) * 2 * NN + r) * NN
                                : p + ((long)(c0 + l) * NN + (r - 2 * NN)) * NN;
      T t[NN], v[NC];
#pragma unroll
      for (int i = 0; i < NN; ++i) t[i] = load_late(row + i);
      eo_interp<K, 1>(t, v);
#pragma unroll
      for (int q = 0; q < NC; ++q) X[l * NF * XS + r * NC + q] = v[q];
    }
  }
  if constexpr (STG) cp_async_wait_all();
  __syncthreads();
  if constexpr (HG && !FB)
    for (int t = tid; t < hlist[0]; t += nt) {
      const int e = hlist[1 + t];
      T o[NN];
      face_C<K, T, true>(w, pfix, pff, mesh, c0 + (e >> 2), e & 3, o);
#pragma unroll
      for (int i = 0; i < NN; ++i) Fs[e * NN + i] = o[i];
    }
  // columns: z-interpolation, fluxes, z-integration; xa and xb replace the
  // column's own x-interpolated values
  {
    const int l = tid / NC, j = tid - l * NC;
    if (l < cnt) {
      T *x = X + l * NF * XS + j;
      T t[NN], wx[NC], wz[NC], V[NC], Gx[NC], Ge[NC];
#pragma unroll
      for (int i = 0; i < NN; ++i) t[i] = x[i * NC];
      eo_interp<K, 1>(t, wx);
#pragma unroll
      for (int i = 0; i < NN; ++i) t[i] = x[XS + i * NC];
      eo_interp<K, 1>(t, wz);
      if (WITH_D) {
        const T *jx = STG ? sJ + (l * NC + j) * NC : mesh.gJ + ((long)(c0 + l) * NC + j) * NC;
#pragma unroll
        for (int i = 0; i < NN; ++i) t[i] = x[2 * XS + i * NC];
        eo_interp<K, 1>(t, V);
#pragma unroll
        for (int q = 0; q < NC; ++q) V[q] *= jx[q];
      }
      const T *h = STG ? sH + (l * NC + j) * NC * 4 : hq + ((long)(c0 + l) * NC + j) * NC * 4;
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        const Vec4<T> H(h + 4 * q, STG ? FROM_SHARED : FROM_LATE);  // (xi, eta) from w_x, then from w_z
        Gx[q] = fma(H.v[0], wx[q], H.v[2] * wz[q]);
        Ge[q] = fma(H.v[1], wx[q], H.v[3] * wz[q]);
      }
      T a[NN], b[NN];
      eo_integ<K, 1, NC, WITH_D, true>(V, Ge, a);
      eo_integ<K, 1, NC, true, false>(Gx, Gx, b);
#pragma unroll
      for (int i = 0; i < NN; ++i) {
        x[i * NC] = a[i];
        x[XS + i * NC] = b[i];
      }
    }
  }
  __syncthreads();
  // output rows: D p - C w
  for (int e = tid; e < cnt * NN; e += nt) {
    const int l = e / NN, iz = e - l * NN;
    const T *x = X + l * NF * XS + iz * NC;
    T a[NC], b[NC], out[NN], add[NN];
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      a[q] = x[q];
      b[q] = x[XS + q];
    }
    eo_integ<K, 1, NC, true, true>(a, b, out);
    if constexpr (FB) face_rows_of<K>(Fb, mesh, c0 + l, iz, add);
    else face_rows<K>(Fs + l * 4 * NN, iz, add);
    const long g0 = (long)(c0 + l) * NN2 + iz * NN;
    T s = cC;
    if (!WITH_D && mesh.dts) s *= mesh.dts[c0 + l];
#pragma unroll
    for (int i = 0; i < NN; ++i) {
      const T r = out[i] - add[i];
      const long g = g0 + i;
      if (MODE == 0) dst[g] = -s * r;
      else if (MODE == 1) dst[g] = r;
      else if (MODE == 2) dst[g] = invd[g] * r;
      else if (MODE == 3) dst[g] += s * r;
      else {
        T rh, iv, dd, xx;
        if constexpr (STG) {
          const T *v = sV + e * NN + i;
          rh = v[0];
          iv = v[cpb * NN2];
          dd = v[2 * cpb * NN2];
          xx = v[3 * cpb * NN2];
        } else {
          rh = ch.rhs[g];
          iv = invd[g];
          dd = ch.d[g];
          xx = ch.x[g];
        }
        const T dk = (ch.first ? T(0) : ch.a * dd) + ch.b * iv * (rh - r);
        ch.d[g] = dk;
        ch.x[g] = xx + dk;
      }
    }
  }
}

// Fb[c][f][k+1]: nodal integrals of C w over the odd local faces, whose conforming
// neighbours read them with the opposite sign, and over both sides of hanging
// faces.
template <int K, typename T, bool HG>
__global__ void __launch_bounds__(64)
    k_exact_face_C(T *__restrict__ Fb, const T *__restrict__ w, const T *__restrict__ pfix,
                   const T *__restrict__ pff, MeshT<T> mesh) {
  constexpr int NN = K + 1;
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  T o[NN];
  int c, f;
  if (!HG || g < 2L * mesh.nc) {  // conforming odd faces
    if (g >= 2L * mesh.nc) return;
    c = (int)(g >> 1);
    f = (int)(g & 1) * 2 + 1;
    if (mesh.nbr[c * 4 + f] < 0 || (HG && (mesh.nbrf[c * 4 + f] >> 2) != 0)) return;
    face_C<K, T, false>(w, pfix, pff, mesh, c, f, o);
  } else {  // hanging faces, each from its own side
    const long e = g - 2L * mesh.nc;
    if (e >= 4L * mesh.nc) return;
    c = (int)(e >> 2);
    f = (int)(e & 3);
    if (mesh.nbr[c * 4 + f] < 0 || (mesh.nbrf[c * 4 + f] >> 2) == 0) return;
    face_C<K, T, true>(w, pfix, pff, mesh, c, f, o);
  }
#pragma unroll
  for (int i = 0; i < NN; ++i) Fb[((long)c * 4 + f) * NN + i] = o[i];
}

// ========================================================== p_fix prep ===
// H = gamma/(gamma-1) p_fix cof at the NC x NC points ([c][qx][qz][4]) and the
// face traces of p_fix at the 2k+1 points.  Threads (cell, column).  Bound by
// its stores at large meshes (1,568 + 288 bytes per cell at k = 4 in FP64).
// `copy` (may be null) receives p_fix itself: on small meshes a launch of its own
// for the copy is 4 us of the 25-75 that freezing rho and p takes (800 cells,
// k = 2: 30.7 -> 26.6 us).
template <int K, typename T>
__global__ void __launch_bounds__(32 * Ex<K>::NC)
    k_exact_pfix(T *__restrict__ hq, T *__restrict__ pff, const T *__restrict__ pfix,
                 T *__restrict__ copy, MeshT<T> mesh, int cpb) {
  using E = Ex<K>;
  constexpr int NN = E::NN, NN2 = E::NN2, NC = E::NC, NQ = E::NQ;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T *X = reinterpret_cast<T *>(sm_raw);  // [cpb][NN][NC]
  const int tid = threadIdx.x, nt = blockDim.x;
  const int c0 = blockIdx.x * cpb;
  const int cnt = min(cpb, mesh.nc - c0);
  for (int e = tid; e < cnt * NN; e += nt) {
    T t[NN], v[NC];
#pragma unroll
    for (int i = 0; i < NN; ++i) t[i] = __ldg(pfix + ((long)c0 * NN + e) * NN + i);
    if (copy) {
#pragma unroll
      for (int i = 0; i < NN; ++i) copy[((long)c0 * NN + e) * NN + i] = t[i];
    }
    eo_interp<K, 1>(t, v);
#pragma unroll
    for (int q = 0; q < NC; ++q) X[e * NC + q] = v[q];
  }
  for (int e = tid; e < cnt * 4; e += nt) {
    T t[NN], v[NQ];
    trace<K>(pfix + (long)(c0 + (e >> 2)) * NN2, e & 3, t);
    eo_interp<K, 2>(t, v);
#pragma unroll
    for (int q = 0; q < NQ; ++q) pff[((long)c0 * 4 + e) * NQ + q] = v[q];
  }
  __syncthreads();
  const int l = tid / NC, j = tid - l * NC;
  if (l >= cnt) return;
  T t[NN], v[NC];
#pragma unroll
  for (int i = 0; i < NN; ++i) t[i] = X[(l * NN + i) * NC + j];
  eo_interp<K, 1>(t, v);
  const long o = ((long)(c0 + l) * NC + j) * NC * 4;
#pragma unroll
  for (int q = 0; q < NC; ++q) {
    Vec4<T> g(mesh.gC + o + 4 * q);
#pragma unroll
    for (int d = 0; d < 4; ++d) g.v[d] *= v[q];
    g.store(hq + o + 4 * q);
  }
}

// ============================================================ launchers ===
// The autotuner's cells per block, rounded up to a multiple of 8 so that the
// face threads of C/D fill whole warps.
inline int exact_cells(int cpb) { return (cpb + 7) / 8 * 8; }

// The modes that are used: FP32 (multigrid levels) B mode 2 and C/D modes 1 and 4;
// FP64 C/D with FB (S and the solver) modes 1, 2 and 3.  Null for the others.
template <int K, typename T, bool HG>
auto exact_B_kernel(int mode) {
  decltype(&k_exact_B<K, 2, T, HG>) fn = mode == 2 ? k_exact_B<K, 2, T, HG> : nullptr;
  if constexpr (sizeof(T) == 8) {
    if (mode == 0) fn = k_exact_B<K, 0, T, HG>;
    if (mode == 1) fn = k_exact_B<K, 1, T, HG>;
  }
  return fn;
}
template <int K, typename T, bool HG>
auto exact_CD_kernel(int mode, bool fb) {
  decltype(&k_exact_CD<K, 1, T, HG, false>) fn = nullptr;
  if constexpr (sizeof(T) == 8) {
    if (fb)
      return mode == 1   ? k_exact_CD<K, 1, T, HG, true>
             : mode == 2 ? k_exact_CD<K, 2, T, HG, true>
             : mode == 3 ? k_exact_CD<K, 3, T, HG, true>
                         : fn;
    if (mode == 0) fn = k_exact_CD<K, 0, T, HG, false>;
    if (mode == 2) fn = k_exact_CD<K, 2, T, HG, false>;
    if (mode == 3) fn = k_exact_CD<K, 3, T, HG, false>;
  }
  if (mode == 1) fn = k_exact_CD<K, 1, T, HG, false>;
  if (mode == 4) fn = k_exact_CD<K, 4, T, HG, false>;
  return fn;
}

template <int K, typename T, bool HG>
int exact_B_launch(const OpView<T> &v, T *dst, const T *p, T cB, T cC, int mode) {
  bool overlap = false;  // not while the tuner times the kernel
  auto launch = [&](int tuned) -> cudaError_t {
    int cpb = v.nc < 2048 ? 8 : exact_cells(tuned);
    if (cpb * ExB<K>::TPC > 320) cpb = 320 / ExB<K>::TPC / 8 * 8;
    const size_t sm =
        sizeof(T) * (size_t)cpb * ExB<K>::template values<T>(mode == 2 && sizeof(T) == 4) +
        (HG ? sizeof(int) * (4 * cpb + 1) : 0);
    auto fn = exact_B_kernel<K, T, HG>(mode);
    if (!fn) return cudaErrorInvalidValue;
    if (cudaError_t e = allow_smem(fn, sm); e != cudaSuccess) return e;
    return launch_overlapped(overlap, fn, (v.nc + cpb - 1) / cpb, cpb * ExB<K>::TPC, sm, v.st, dst, p, cB,
                             cC, v.ainv, v.mesh, cpb);
  };
  // mode 1 (dst -= B p) is not idempotent: it uses the choice made for mode 0
  const int cpb = tuned_cpb(v.tune, v.st, TF_B, K, mode == 1 ? 0 : mode, HG, (int)sizeof(T),
                            v.nc, mode != 1 && dst != p, launch);
  overlap = !HG;
  ATM_CUDA(launch(cpb));
  g_kernel_launches.fetch_add(1);
  return ATM_OK;
}

template <int K, typename T, bool HG>
int exact_CD_launch(const OpView<T> &v, T *dst, const T *w, const T *p, T cC, int mode,
                    const ChebArgs<T> *cheb) {
  using E = Ex<K>;
  const T *pfix = v.pfix;
  const ChebArgs<T> ch = cheb ? *cheb : ChebArgs<T>{};
  const bool fb = sizeof(T) == 8 && v.fbuf;
  bool overlap = false;  // not while the tuner times the kernel
  auto launch = [&](int tuned) -> cudaError_t {
    int cpb = v.nc < 2048 ? 8 : exact_cells(tuned);
    if (cpb > 32) cpb = 32;
    // FB: the tuner's candidates are 64, 128 and 256 threads' worth of columns
    if (fb) cpb = (tuned >= 256 / E::NQ ? 256 : tuned >= 128 / E::NQ ? 128 : 64) / E::NC;
    const int staged = sizeof(T) == 4 ? 5 * E::NC2 + (mode == 4 ? 4 * E::NN2 : 0) : 0;
    const size_t sm = sizeof(T) * (size_t)cpb *
                      ((mode == 0 || mode == 3 ? 2 : 3) * E::NN * E::NC + 4 * E::NN + staged) +
                      (HG ? sizeof(int) * (4 * cpb + 1) : 0);
    auto fn = exact_CD_kernel<K, T, HG>(mode, fb);
    if (!fn) return cudaErrorInvalidValue;
    if (cudaError_t e = allow_smem(fn, sm); e != cudaSuccess) return e;
    return launch_overlapped(overlap, fn, (v.nc + cpb - 1) / cpb, cpb * E::NC, sm, v.st, dst, w, p,
                             pfix, v.pfq, v.pff, (const T *)v.fbuf, cC, v.invd, v.mesh, ch, cpb);
  };
  if constexpr (sizeof(T) == 8)
    if (fb) {
      const long n = (long)v.nc * (HG ? 6 : 2);
      k_exact_face_C<K, T, HG><<<(unsigned)((n + 63) / 64), 64, 0, v.st>>>(v.fbuf, w, pfix, v.pff,
                                                                         v.mesh);
      ATM_CHECK_LAUNCH("k_exact_face_C");
    }
  // modes 3 (dst -= C w) and 4 (x += d) are not idempotent: they use the
  // choices made for modes 0 and 1
  const bool idem = mode < 3 && dst != w && dst != p && dst != pfix;
  const int key = mode == 3 ? 0 : (mode == 4 ? 1 : mode);
  const int cpb = tuned_cpb(v.tune, v.st, fb ? TF_CD_FACES : TF_CD, K, key, HG, (int)sizeof(T),
                            v.nc, idem, launch);
  overlap = !HG && !fb;
  ATM_CUDA(launch(cpb));
  g_kernel_launches.fetch_add(1);
  return ATM_OK;
}

// p_fix from `src` (also copied to v.pfix when that is another vector)
template <int K, typename T>
int exact_pfix_launch(const OpView<T> &v, const T *src) {
  using E = Ex<K>;
  const int cpb = v.nc < 4096 ? 8 : 32;
  k_exact_pfix<K, T><<<(v.nc + cpb - 1) / cpb, cpb * E::NC, sizeof(T) * cpb * E::NN * E::NC, v.st>>>(
      const_cast<T *>(v.pfq), const_cast<T *>(v.pff), src,
      src == v.pfix ? nullptr : const_cast<T *>(v.pfix), v.mesh, cpb);
  ATM_CHECK_LAUNCH("k_exact_pfix");
  return ATM_OK;
}

}  // namespace atm
