// Device and launch helpers that need no basis tables: the layout of the
// A^{-1} blocks, asynchronous copies, the shared-memory limit.
#pragma once
#include "atm_internal.h"

namespace atm {

// source vectors of a right-hand side, in the operator's positional order
struct SrcPtrs {
  const double *p[12];
};

// max(|a|, |b|) on the integer pipe for doubles (a double comparison takes an
// FP64 issue slot); a NaN on either side gives a NaN
__device__ __forceinline__ double abs_max(double a, double b) {
  const long long m = 0x7fffffffffffffffll;
  const long long x = __double_as_longlong(a) & m, y = __double_as_longlong(b) & m;
  return __longlong_as_double(x > y ? x : y);
}
__device__ __forceinline__ float abs_max(float a, float b) {
  const int m = 0x7fffffff;
  const int x = __float_as_int(a) & m, y = __float_as_int(b) & m;
  return __int_as_float(x > y ? x : y);
}

// Values between two cells' A^{-1} blocks ([nc][stride]).  FP64: the full
// (k+1)^2 x (k+1)^2 block.  FP32 (multigrid levels): A^{-1} is symmetric, so
// only its lower triangle is stored, for the general kernels row by row ((r, c <= r)
// at r (r+1)/2 + c, padded to a multiple of four values) and for the `exact` ones
// as (k+1) x (k+1) tiles: tile (a, b), b <= a,
// couples the node rows iz = a and iz = b.  Off-diagonal tiles come first
// (row by row, each padded to a multiple of four values), then the diagonal
// ones as packed lower triangles.  The B kernel stages the blocks of its cells
// into shared memory with 16-byte copies and reads tiles in 16-byte loads; the
// stride is 4 mod 8 values, so that eight cells' equal offsets fall into
// eight different groups of four banks.
template <int K>
struct ATile {
  static constexpr int NN = K + 1;
  static constexpr int OFF = (NN * NN + 3) / 4 * 4;               // an off-diagonal tile
  static constexpr int DIA = (NN * (NN + 1) / 2 + 3) / 4 * 4;     // a diagonal tile
  static constexpr int D0 = NN * (NN - 1) / 2 * OFF;              // first diagonal tile
  static constexpr int USED = D0 + NN * DIA;
  static constexpr int STRIDE = USED % 8 == 4 ? USED : USED + 4;
};
template <int K, typename T>
__host__ __device__ constexpr int ainv_stride(bool exact = true) {
  constexpr int N2 = (K + 1) * (K + 1);
  return sizeof(T) == 8 ? N2 * N2 : exact ? ATile<K>::STRIDE : (N2 * (N2 + 1) / 2 + 3) / 4 * 4;
}
// offset of entry (i, j), i >= j, in the FP32 tiles
template <int K>
__device__ __forceinline__ int atile_index(int i, int j) {
  constexpr int NN = K + 1;
  const int a = i / NN, b = j / NN, r = i - a * NN, c = j - b * NN;
  if (a == b) return ATile<K>::D0 + a * ATile<K>::DIA + r * (r + 1) / 2 + c;
  return (a * (a - 1) / 2 + b) * ATile<K>::OFF + r * NN + c;
}
inline long ainv_stride_rt(int k, size_t elem, bool exact) {
  if (elem != 4) return (long)(k + 1) * (k + 1) * (k + 1) * (k + 1);
  switch (k) {
    case 1: return ainv_stride<1, float>(exact);
    case 2: return ainv_stride<2, float>(exact);
    case 3: return ainv_stride<3, float>(exact);
    case 4: return ainv_stride<4, float>(exact);
    default: return ainv_stride<5, float>(exact);
  }
}

// 16-byte asynchronous global -> shared copies (cp.async, bypassing L1) and
// the wait for all of this thread's outstanding copies
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Programmatic dependent launch: a kernel launched by launch_overlapped may
// become resident while its predecessor in the stream drains, so that launch
// latency and the predecessor's tail overlap.  Such a kernel calls
// pdl_trigger() (its own successor may do the same) and must call pdl_wait()
// before it touches anything that an overlapped kernel or the launch directly
// before it writes or reads: the wait returns when the predecessor, and with it
// everything before, has completed.  What earlier launches wrote may be read
// sooner, provided that at least one kernel launched without overlap lies between
// (it started after they had completed, and this one starts after it).
// Values that the launch directly before may have written are loaded with
// load_late: the read-only path (__ldg, const __restrict__) is for data that nobody
// writes during the kernel's lifetime, which begins before the wait.
// A kernel triggers only if its successor's blocks then spread well: early
// blocks of a grid that fits the GPU in a wave pack the SMs that are free first.
// C/D does not trigger: the next operator's B packed itself that way and S took
// 307 instead of 249 us at 11,781 cells, k = 5.  Not inside a stream capture
// (replayed V-cycle graphs got 7% slower with programmatic edges) and not for
// the hanging-face kernels (6300 cells, k = 3: 84 -> 88 us).  Elsewhere S takes
// 18.4 instead of 22.5 us at 800 cells, k = 2, 249 instead of 252 at 11,781, k = 5.
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ double load_late(const double *p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ float load_late(const float *p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
template <typename... P, typename... A>
inline cudaError_t launch_overlapped(bool overlap, void (*fn)(P...), long grid, int block, size_t smem,
                                     cudaStream_t st, A... args) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) {
    cudaGetLastError();
    overlap = false;
  }
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = overlap && cap == cudaStreamCaptureStatusNone ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, fn, P(args)...);
}

// Let kernel `fn` use up to the device's opt-in maximum of dynamic shared
// memory when a launch needs more than the default 48 KB.  The limit is set
// to that maximum, always the same value: host threads launching the same
// kernel with different block shapes (serving members, the autotuner) must
// never lower each other's limit between setting it and launching.
template <typename F>
inline cudaError_t allow_smem(F fn, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  static int cap[64] = {0};  // per device; a benign race writes the same value
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int mx = dev >= 0 && dev < 64 ? cap[dev] : 0;
  if (mx == 0) {
    e = cudaDeviceGetAttribute(&mx, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) cap[dev] = mx;
  }
  if (bytes > (size_t)mx) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
}

}  // namespace atm
