// FP64 instantiations of the Schur kernels for mappings of degree <= 2 on 2:1
// adaptive meshes (hanging faces).
#include "schur_exact.cuh"

namespace atm {

int upload_exact_hang(const double *t) { return upload_exact_here(t); }

int exact_B_hang(const OpView<double> &o, double *dst, const double *p, double cB, double cC, int mode) {
  ATM_DISPATCH_K(o.k, (exact_B_launch<K, double, true>(o, dst, p, cB, cC, mode)));
}
int exact_CD_hang(const OpView<double> &o, double *dst, const double *w, const double *p, double cC, int mode,
                  const ChebArgs<double> *ch) {
  ATM_DISPATCH_K(o.k, (exact_CD_launch<K, double, true>(o, dst, w, p, cC, mode, ch)));
}

}  // namespace atm
