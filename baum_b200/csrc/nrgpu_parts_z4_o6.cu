// nrgpu_parts_z4_o6.cu -- the two rhs kernels for Z4c, order 6.
#include "nrgpu_parts.cuh"

void nrgpu_z4_parts_o6(nrgpu_level *L, const RhsWork &w, int b, const double *const *U, double *const *out,
                       const double *const *pre, double *const *acc, const Epilogue &E, const nrgpu_z4_params &p,
                       cudaStream_t st, int kb, int ke) {
  launch_parts<NRGPU_Z4_NVARS, 6>(L, w, b, U, out, pre, acc, E, p, st, kb, ke);
}
