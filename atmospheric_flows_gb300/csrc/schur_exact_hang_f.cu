// FP32 instantiations of the Schur kernels for mappings of degree <= 2 on 2:1
// adaptive meshes (hanging faces).
#include "schur_exact.cuh"

namespace atm {

int upload_exact_hang_f(const double *t) { return upload_exact_here(t); }

int exact_B_hang(const OpView<float> &o, float *dst, const float *p, float cB, float cC, int mode) {
  ATM_DISPATCH_K(o.k, (exact_B_launch<K, float, true>(o, dst, p, cB, cC, mode)));
}
int exact_CD_hang(const OpView<float> &o, float *dst, const float *w, const float *p, float cC, int mode,
                  const ChebArgs<float> *ch) {
  ATM_DISPATCH_K(o.k, (exact_CD_launch<K, float, true>(o, dst, w, p, cC, mode, ch)));
}

}  // namespace atm
