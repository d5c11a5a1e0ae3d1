// 1D contractions shared by the operator kernels.  One thread contracts a whole
// row, column or face trace: the coefficients are compile-time constant-bank
// operands and the even-odd split of the symmetric point sets applies (Gauss
// and Gauss-Lobatto points: S(P-1-q, k-i) = S(q, i), D(P-1-q, k-i) = -D(q, i)).
// FP64 instructions are what these kernels pay for (two lanes per clock and SM
// on sm_103a); a contraction of k+1 values to P points takes 28 instead of 35
// of them for k = 4, P = 7.
#pragma once
#include "device_util.cuh"

namespace atm {

template <int K>
struct Ex {
  static constexpr int NN = K + 1, NN2 = NN * NN;
  static constexpr int NQ = 2 * K + 1;         // face points of C
  static constexpr int NC = (3 * K + 3) / 2;   // volume points per direction of C and D
  static constexpr int NC2 = NC * NC;
};

// Even-odd halves of the 1D tables of one point set: [kind][q][i] for
// q < ceil(NP/2), i < ceil(NN/2), kind 0 E_S, 1 O_S, 2 E_D, 3 O_D with
// E = (M(q,i) + M(q,k-i)) / 2 and O = (M(q,i) - M(q,k-i)) / 2.  Sets: 0 the
// k+1, 1 the NC, 2 the 2k+1 Gauss points.
constexpr int EO_Q = 6, EO_I = 3, EO_SETS = 3;
static __constant__ double c_eo[KMAX + 1][EO_SETS][4][EO_Q][EO_I];
static __constant__ float c_eo_f[KMAX + 1][EO_SETS][4][EO_Q][EO_I];
// basis values at the subface points (g_q + s)/2 of hanging faces:
// [k][0: the k+1 points, 1: the 2k+1 points][s][q][i]
static __constant__ double c_sub[KMAX + 1][2][2][NQ_MAX][NN_MAX];
static __constant__ float c_sub_f[KMAX + 1][2][2][NQ_MAX][NN_MAX];
constexpr int EO_DOUBLES = (KMAX + 1) * EO_SETS * 4 * EO_Q * EO_I;
constexpr int SUB_DOUBLES = (KMAX + 1) * 4 * NQ_MAX * NN_MAX;

// `table`: c_eo followed by c_sub (upload_exact_all)
static inline int upload_exact_here(const double *table) {
  std::vector<float> f(table, table + EO_DOUBLES + SUB_DOUBLES);
  if (cudaMemcpyToSymbol(c_eo, table, sizeof(c_eo)) != cudaSuccess) return 1;
  if (cudaMemcpyToSymbol(c_sub, table + EO_DOUBLES, sizeof(c_sub)) != cudaSuccess) return 1;
  if (cudaMemcpyToSymbol(c_eo_f, f.data(), sizeof(c_eo_f)) != cudaSuccess) return 1;
  return cudaMemcpyToSymbol(c_sub_f, f.data() + EO_DOUBLES, sizeof(c_sub_f)) == cudaSuccess ? 0 : 1;
}

template <typename T>
struct CEo;
template <>
struct CEo<double> {
  static __device__ __forceinline__ double get(int k, int s, int w, int q, int i) {
    return c_eo[k][s][w][q][i];
  }
  static __device__ __forceinline__ double sub(int k, int p, int s, int q, int i) {
    return c_sub[k][p][s][q][i];
  }
};
template <>
struct CEo<float> {
  static __device__ __forceinline__ float get(int k, int s, int w, int q, int i) {
    return c_eo_f[k][s][w][q][i];
  }
  static __device__ __forceinline__ float sub(int k, int p, int s, int q, int i) {
    return c_sub_f[k][p][s][q][i];
  }
};

// v_q = sum_i S(q,i) t_i
template <int K, int SET, int NP, typename T>
__device__ __forceinline__ void eo_interp(const T (&t)[K + 1], T (&v)[NP]) {
  constexpr int H = (K + 1) / 2, P = NP / 2;
  constexpr bool MI = ((K + 1) & 1) != 0, MQ = (NP & 1) != 0;
  T te[H], to[H];
#pragma unroll
  for (int i = 0; i < H; ++i) {
    te[i] = t[i] + t[K - i];
    to[i] = t[i] - t[K - i];
  }
#pragma unroll
  for (int q = 0; q < P; ++q) {
    T e = CEo<T>::get(K, SET, 0, q, 0) * te[0], o = CEo<T>::get(K, SET, 1, q, 0) * to[0];
#pragma unroll
    for (int i = 1; i < H; ++i) {
      e = fma(CEo<T>::get(K, SET, 0, q, i), te[i], e);
      o = fma(CEo<T>::get(K, SET, 1, q, i), to[i], o);
    }
    if (MI) e = fma(CEo<T>::get(K, SET, 0, q, H), t[H], e);
    v[q] = e + o;
    v[NP - 1 - q] = e - o;
  }
  if (MQ) {
    T e = CEo<T>::get(K, SET, 0, P, 0) * te[0];
#pragma unroll
    for (int i = 1; i < H; ++i) e = fma(CEo<T>::get(K, SET, 0, P, i), te[i], e);
    if (MI) e = fma(CEo<T>::get(K, SET, 0, P, H), t[H], e);
    v[P] = e;
  }
}

// v_q = sum_i S(q,i) t_i and d_q = sum_i D(q,i) t_i
template <int K, int SET, int NP, typename T>
__device__ __forceinline__ void eo_interp_d(const T (&t)[K + 1], T (&v)[NP], T (&d)[NP]) {
  constexpr int H = (K + 1) / 2, P = NP / 2;
  constexpr bool MI = ((K + 1) & 1) != 0, MQ = (NP & 1) != 0;
  eo_interp<K, SET>(t, v);
  T te[H], to[H];
#pragma unroll
  for (int i = 0; i < H; ++i) {
    te[i] = t[i] + t[K - i];
    to[i] = t[i] - t[K - i];
  }
#pragma unroll
  for (int q = 0; q < P + (MQ ? 1 : 0); ++q) {
    T b = CEo<T>::get(K, SET, 3, q, 0) * to[0];
#pragma unroll
    for (int i = 1; i < H; ++i) b = fma(CEo<T>::get(K, SET, 3, q, i), to[i], b);
    if (MQ && q == P) {  // E_D = 0 at the middle point
      d[P] = b;
    } else {
      T a = CEo<T>::get(K, SET, 2, q, 0) * te[0];
#pragma unroll
      for (int i = 1; i < H; ++i) a = fma(CEo<T>::get(K, SET, 2, q, i), te[i], a);
      if (MI) a = fma(CEo<T>::get(K, SET, 2, q, H), t[H], a);
      d[q] = b + a;
      d[NP - 1 - q] = b - a;
    }
  }
}
// d_q = sum_i D(q,i) t_i alone
template <int K, int SET, int NP, typename T>
__device__ __forceinline__ void eo_deriv(const T (&t)[K + 1], T (&d)[NP]) {
  T v[NP];
  eo_interp_d<K, SET>(t, v, d);  // the unused values are dropped by the compiler
}

// out_i = sum_q S(q,i) V_q + D(q,i) G_q
template <int K, int SET, int NP, bool HAS_V, bool HAS_G, typename T>
__device__ __forceinline__ void eo_integ(const T (&V)[NP], const T (&G)[NP], T (&out)[K + 1]) {
  static_assert(HAS_V || HAS_G, "nothing to integrate");
  constexpr int H = (K + 1) / 2, P = NP / 2;
  constexpr bool MI = ((K + 1) & 1) != 0, MQ = (NP & 1) != 0;
  T ve[P], vo[P], ge[P], go[P];
#pragma unroll
  for (int q = 0; q < P; ++q) {
    if (HAS_V) {
      ve[q] = V[q] + V[NP - 1 - q];
      vo[q] = V[q] - V[NP - 1 - q];
    }
    if (HAS_G) {
      ge[q] = G[q] + G[NP - 1 - q];
      go[q] = G[q] - G[NP - 1 - q];
    }
  }
#pragma unroll
  for (int i = 0; i < H; ++i) {
    T e = HAS_V ? CEo<T>::get(K, SET, 0, 0, i) * ve[0] : CEo<T>::get(K, SET, 2, 0, i) * go[0];
    T o = HAS_V ? CEo<T>::get(K, SET, 1, 0, i) * vo[0] : CEo<T>::get(K, SET, 3, 0, i) * ge[0];
    if (HAS_V && HAS_G) {
      e = fma(CEo<T>::get(K, SET, 2, 0, i), go[0], e);
      o = fma(CEo<T>::get(K, SET, 3, 0, i), ge[0], o);
    }
#pragma unroll
    for (int q = 1; q < P; ++q) {
      if (HAS_V) {
        e = fma(CEo<T>::get(K, SET, 0, q, i), ve[q], e);
        o = fma(CEo<T>::get(K, SET, 1, q, i), vo[q], o);
      }
      if (HAS_G) {
        e = fma(CEo<T>::get(K, SET, 2, q, i), go[q], e);
        o = fma(CEo<T>::get(K, SET, 3, q, i), ge[q], o);
      }
    }
    if (MQ && HAS_V) e = fma(CEo<T>::get(K, SET, 0, P, i), V[P], e);
    if (MQ && HAS_G) o = fma(CEo<T>::get(K, SET, 3, P, i), G[P], o);
    out[i] = e + o;
    out[K - i] = e - o;
  }
  if (MI) {  // i = k/2: O_S = O_D = 0 and D(mid, k/2) = 0
    T e = HAS_V ? CEo<T>::get(K, SET, 0, 0, H) * ve[0] : CEo<T>::get(K, SET, 2, 0, H) * go[0];
    if (HAS_V && HAS_G) e = fma(CEo<T>::get(K, SET, 2, 0, H), go[0], e);
#pragma unroll
    for (int q = 1; q < P; ++q) {
      if (HAS_V) e = fma(CEo<T>::get(K, SET, 0, q, H), ve[q], e);
      if (HAS_G) e = fma(CEo<T>::get(K, SET, 2, q, H), go[q], e);
    }
    if (MQ && HAS_V) e = fma(CEo<T>::get(K, SET, 0, P, H), V[P], e);
    out[H] = e;
  }
}

// how four values are loaded: from a table that does not change, from shared
// memory, or (FP64) from global memory that the launch before may have written
enum LoadFrom { FROM_TABLE, FROM_SHARED, FROM_LATE };
template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
  float v[4];
  __device__ __forceinline__ explicit Vec4(const float *p, LoadFrom from = FROM_TABLE) {  // 16-byte aligned
    const float4 *s = reinterpret_cast<const float4 *>(p);
    const float4 a = from == FROM_SHARED ? *s : __ldg(s);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  }
  __device__ __forceinline__ void store(float *p) const {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
};
template <>
struct Vec4<double> {
  double v[4];
  __device__ __forceinline__ explicit Vec4(const double *p, LoadFrom from = FROM_TABLE) {  // 16-byte aligned
    if (from == FROM_LATE) {
#pragma unroll
      for (int i = 0; i < 4; i += 2)
        asm volatile("ld.global.v2.f64 {%0, %1}, [%2];"
                     : "=d"(v[i]), "=d"(v[i + 1])
                     : "l"(__cvta_generic_to_global(p + i)));
    } else {
      const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
      const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
  }
  __device__ __forceinline__ void store(double *p) const {
    reinterpret_cast<double2 *>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2 *>(p)[1] = make_double2(v[2], v[3]);
  }
};
__device__ __forceinline__ void load2(const float *p, float &a, float &b) {  // 8-byte aligned
  const float2 x = __ldg(reinterpret_cast<const float2 *>(p));
  a = x.x; b = x.y;
}
__device__ __forceinline__ void load2(const double *p, double &a, double &b) {  // 16-byte
  const double2 x = __ldg(reinterpret_cast<const double2 *>(p));
  a = x.x; b = x.y;
}

// nodal trace of a cell's field on face f (LATE: load_late)
template <int K, bool LATE = false, typename T>
__device__ __forceinline__ void trace(const T *__restrict__ cell, int f, T (&t)[K + 1]) {
  constexpr int NN = K + 1;
  const T *b = cell + (f == 1 ? K : f == 3 ? K * NN : 0);
  const int st = f < 2 ? NN : 1;
#pragma unroll
  for (int i = 0; i < NN; ++i) t[i] = LATE ? load_late(b + i * st) : __ldg(b + i * st);
}
// the same trace at the points of subface s (point set PS: 0 k+1, 1 2k+1)
template <int K, int PS, int NP, typename T>
__device__ __forceinline__ void sub_interp(const T (&t)[K + 1], int s, T (&v)[NP]) {
  for (int q = 0; q < NP; ++q) {
    T a = CEo<T>::sub(K, PS, s, q, 0) * t[0];
#pragma unroll
    for (int i = 1; i <= K; ++i) a = fma(CEo<T>::sub(K, PS, s, q, i), t[i], a);
    v[q] = a;
  }
}
template <int K, int PS, int NP, typename T>
__device__ __forceinline__ void sub_integ_add(const T (&F)[NP], int s, T (&out)[K + 1]) {
#pragma unroll
  for (int i = 0; i <= K; ++i)
    for (int q = 0; q < NP; ++q) out[i] = fma(CEo<T>::sub(K, PS, s, q, i), F[q], out[i]);
}

// trace of a cell's field at the 2k+1 points of face f (sub < 0) or of its
// subface `sub`
template <int K, int NP, typename T>
__device__ __forceinline__ void own_or_sub(const T *__restrict__ cell, int f, int sub, T (&v)[NP]) {
  T t[K + 1];
  trace<K>(cell, f, t);
  if (sub < 0) eo_interp<K, 2>(t, v);
  else sub_interp<K, 1>(t, sub, v);
}

}  // namespace atm
