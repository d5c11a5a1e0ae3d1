// FP32 instantiations of the general Schur kernels B and C/D (mapping degree >= 3)
// for the levels of the mixed-precision multigrid on conforming meshes.  A
// translation unit of its own: compiled together with impl_kernels.cu, the C/D
// kernel of k = 4 came out with 168 bytes of spills at the same 64 registers (FP32
// V-cycle of 160x80, mapping degree 3: 0.69 instead of 0.63 ms).
#include "schur_kernels.cuh"

namespace atm {

int upload_basis_general_f(const double *t) { return upload_basis_here(t); }

int general_B_f(const OpView<float> &o, float *dst, const float *p, float cB) {
  ATM_DISPATCH_K(o.k, (B_launch<K, float, false>(o, dst, p, cB, 2)));
}
int general_CD_f(const OpView<float> &o, float *dst, const float *w, const float *p, float cC,
                 int mode, const ChebArgs<float> *ch) {
  ATM_DISPATCH_K(o.k, (CD_launch<K, float, false>(o, dst, w, p, cC, mode, ch)));
}

}  // namespace atm
