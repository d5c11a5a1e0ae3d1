// Face kernels of the explicit right-hand sides on 2:1 adaptive meshes
// (rhs_kernels.cuh), apart from the conforming ones so that they compile in
// parallel.
#include "rhs_kernels.cuh"

namespace atm {

int upload_contract_hang_rhs(const double *t) { return upload_exact_here(t); }

int rhs_face_hang(const atm_ctx &c, int kind, int stage, double *dst, int way, const SrcPtrs &sp,
                  const StageCoef &co) {
  switch (kind) {
    case 0: return rhs_face_dispatch<0, true>(c, stage, dst, way, sp, co);
    case 1: return rhs_face_dispatch<1, true>(c, stage, dst, way, sp, co);
    default: return rhs_face_dispatch<2, true>(c, stage, dst, way, sp, co);
  }
}

}  // namespace atm
