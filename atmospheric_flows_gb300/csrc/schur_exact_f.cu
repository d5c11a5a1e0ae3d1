// FP32 instantiations of the Schur kernels for mappings of degree <= 2 on
// conforming multigrid levels (a translation unit of its own so that it
// compiles in parallel with the others).
#include "schur_exact.cuh"

namespace atm {

int upload_exact_f(const double *t) { return upload_exact_here(t); }

int exact_B_hang(const OpView<float> &o, float *dst, const float *p, float cB, float cC, int mode);
int exact_CD_hang(const OpView<float> &o, float *dst, const float *w, const float *p, float cC,
                  int mode, const ChebArgs<float> *ch);

int exact_B(const OpView<float> &o, float *dst, const float *p, float cB, float cC, int mode) {
  if (o.mesh.nhang > 0) return exact_B_hang(o, dst, p, cB, cC, mode);
  ATM_DISPATCH_K(o.k, (exact_B_launch<K, float, false>(o, dst, p, cB, cC, mode)));
}
int exact_CD(const OpView<float> &o, float *dst, const float *w, const float *p, float cC,
             int mode, const ChebArgs<float> *ch) {
  if (o.mesh.nhang > 0) return exact_CD_hang(o, dst, w, p, cC, mode, ch);
  ATM_DISPATCH_K(o.k, (exact_CD_launch<K, float, false>(o, dst, w, p, cC, mode, ch)));
}
int exact_pfix(const OpView<float> &o, const float *src) {
  ATM_DISPATCH_K(o.k, (exact_pfix_launch<K, float>(o, src)));
}

}  // namespace atm
