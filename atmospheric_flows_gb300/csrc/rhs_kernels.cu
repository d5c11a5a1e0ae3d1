// Explicit IMEX stage right-hand sides: the cell kernels, the face kernels of
// conforming meshes and the public launchers (rhs_kernels.cuh).
#include "rhs_kernels.cuh"

namespace atm {

int upload_contract_rhs(const double *t) { return upload_exact_here(t); }

// face kernels of meshes with hanging faces (hang_rhs.cu)
int rhs_face_hang(const atm_ctx &c, int kind, int stage, double *dst, int way, const SrcPtrs &sp,
                  const StageCoef &co);

namespace {
template <int K, int KIND>
int rhs_passes(const atm_ctx &c, int stage, double *dst, const SrcPtrs &sp, const StageCoef &co,
               bool aliased) {
  using E = Ex<K>;
  const bool ex = KIND == 0 && c.mesh.exact;
  const int np = ex ? E::NC : E::NQ;
  const bool held = !aliased;
  void (*fn)(double *, SrcPtrs, StageCoef, Mesh, bool, int);
  if (ex) {
    constexpr bool X = KIND == 0;
    fn = stage == 1 ? k_rhs_cell<K, 1, KIND, X>
                    : (stage == 2 ? k_rhs_cell<K, 2, KIND, X> : k_rhs_cell<K, 3, KIND, X>);
  } else {
    fn = stage == 1 ? k_rhs_cell<K, 1, KIND, false>
                    : (stage == 2 ? k_rhs_cell<K, 2, KIND, false> : k_rhs_cell<K, 3, KIND, false>);
  }
  auto launch = [&](int tuned) -> cudaError_t {
    // the tuner's candidates are 64, 128 and 256 threads' worth of columns;
    // below 2048 cells it has no say: small blocks reach more SMs
    const int threads = tuned >= 256 / E::NQ ? 256 : (tuned >= 128 / E::NQ ? 128 : 64);
    const int cpb = (c.nc < 2048 ? 64 : threads) / np;
    const size_t sm = sizeof(double) * (size_t)cpb *
                      (RhsKind<KIND>::NF * E::NN * np + (held ? RhsKind<KIND>::NCOMP * FACE_VALUES<K> : 0));
    if (cudaError_t e = allow_smem(fn, sm); e != cudaSuccess) return e;
    fn<<<(c.nc + cpb - 1) / cpb, cpb * np, sm, c.stream>>>(dst, sp, co, c.mesh, held, cpb);
    return cudaGetLastError();
  };
  auto faces = [&](int way) {
    return c.mesh.nhang > 0 ? rhs_face_hang(c, KIND, stage, dst, way, sp, co)
                            : rhs_face_launch<K, KIND, false>(c, stage, dst, way, sp, co);
  };
  // the tuner runs the cell kernel on whatever dst holds, before the faces fill it
  const int family = KIND == 0 && !ex ? TF_RHS_RHO_GENERAL : TF_RHS_RHO + KIND;
  const int cpb = tuned_cpb(c.autotune && !c.capturing, c.stream, family, K, stage,
                            c.mesh.nhang > 0, 8, c.nc, !aliased, launch);
  if (held) {
    if (!FACE_SLOTS<K>)
      ATM_CUDA(cudaMemsetAsync(dst, 0, RhsKind<KIND>::NCOMP * c.n_scalar() * sizeof(double), c.stream));
    if (int rc = faces(FACE_HELD)) return rc;
  }
  ATM_CUDA(launch(cpb));
  g_kernel_launches.fetch_add(1);
  if (held) return ATM_OK;
  if (int rc = faces(FACE_ADD_X)) return rc;
  return faces(FACE_ADD_Z);
}

template <int KIND>
int rhs_launch(const atm_ctx &c, int stage, double *dst, const double *const *src,
               const StageCoef &co) {
  if (stage < 1 || stage > 3) return ATM_BAD_ARG;
  SrcPtrs sp{};
  int nsrc;
  rhs_sources(sp, nsrc, KIND, stage, src);
  // dst may overlap a source that only the cell kernel reads
  bool aliased = false;
  for (int i = 0; i < nsrc; ++i) {
    const bool velocity = i % RhsKind<KIND>::PER == 1;
    const uintptr_t a = (uintptr_t)src[i], d = (uintptr_t)dst;
    aliased = aliased || (a < d + RhsKind<KIND>::NCOMP * c.n_scalar() * sizeof(double) &&
                          d < a + (velocity ? 2 : 1) * c.n_scalar() * sizeof(double) && src[i]);
  }
  // algorithmic bytes: every source field read once, the result written once
  const int k = c.k, nout = KIND == 1 ? 2 : 1;
  const int nfields =
      KIND == 0 ? 3 * stage : (KIND == 1 ? 4 * stage + (stage < 3) : 4 * stage + 3);
  const double bytes = 8.0 * c.nc * c.nn2 * (nfields + nout);
  // contractions: evaluate every source field, integrate values and gradients
  // per output component, the traces of both sides and the integration of two
  // faces per cell
  const int ntrace = (KIND == 0 ? 3 : 4) * stage;
  const double flops = c.nc * (nfields * fl_eval(k) + nout * fl_integrate(k, true) +
                               2.0 * (2 * ntrace * fl_face(k) + nout * fl_face(k)));
  TimedRegion tr(c, KF_RHS_RHO + KIND, bytes, flops);
  ATM_DISPATCH_K(k, (rhs_passes<K, KIND>(c, stage, dst, sp, co, aliased)));
}
}  // namespace

int launch_rhs_rho(const atm_ctx &c, int stage, double *dst, const double *const *src,
                   const StageCoef &co) {
  return rhs_launch<0>(c, stage, dst, src, co);
}
int launch_rhs_vel(const atm_ctx &c, int stage, double *dst, const double *const *src,
                   const StageCoef &co) {
  return rhs_launch<1>(c, stage, dst, src, co);
}
int launch_rhs_pres(const atm_ctx &c, int stage, double *dst, const double *const *src,
                    const StageCoef &co) {
  return rhs_launch<2>(c, stage, dst, src, co);
}

namespace {
template <int K>
int rhs_kinetic_launch(const atm_ctx &c, double *dst, const double *base, const double *rho,
                       const double *u, double wgrav, double M2) {
  constexpr int NP = 2 * K + 1;
  const int cpb = (c.nc < 2048 ? 64 : 128) / NP;
  const size_t sm = sizeof(double) * (size_t)cpb * 3 * (K + 1) * NP;
  ATM_CUDA(allow_smem(k_rhs_kinetic<K>, sm));
  k_rhs_kinetic<K><<<(c.nc + cpb - 1) / cpb, cpb * NP, sm, c.stream>>>(dst, base, rho, u, wgrav, M2,
                                                                     c.mesh, cpb);
  ATM_CHECK_LAUNCH("k_rhs_kinetic");
  return ATM_OK;
}
}  // namespace

int launch_rhs_kinetic(const atm_ctx &c, int stage, double *dst, const double *base,
                       const double *rho, const double *u, const StageCoef &co) {
  const double M2 = co.Ma * co.Ma;
  const double wgrav = stage < 3 ? co.cg[stage] * co.dt * M2 / (co.Fr * co.Fr) : 0.0;
  TimedRegion tr(c, KF_RHS_PRES, 8.0 * c.nc * c.nn2 * 5,
                 c.nc * (3 * fl_eval(c.k) + fl_integrate(c.k, false)));
  ATM_DISPATCH_K(c.k, (rhs_kinetic_launch<K>(c, dst, base, rho, u, wgrav, M2)));
}

}  // namespace atm
