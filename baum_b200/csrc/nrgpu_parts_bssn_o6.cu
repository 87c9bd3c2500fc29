// nrgpu_parts_bssn_o6.cu -- the two rhs kernels for BSSN, order 6.
#include "nrgpu_parts.cuh"

void nrgpu_bssn_parts_o6(nrgpu_level *L, const RhsWork &w, int b, const double *const *U, double *const *out,
                         const double *const *pre, double *const *acc, const Epilogue &E, const nrgpu_bssn_params &p,
                         cudaStream_t st, int kb, int ke) {
  launch_parts<NRGPU_NV, 6>(L, w, b, U, out, pre, acc, E, p, st, kb, ke);
}
