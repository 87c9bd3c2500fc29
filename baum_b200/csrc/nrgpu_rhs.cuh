// nrgpu_rhs.cuh -- what the right-hand-side kernels of both systems share:
// variable numbers, lopsided advection rows, Kreiss-Oliger sums, prefetch
// hints and the algebraic constraints of an updated point.
#pragma once
#include "nrgpu_level.cuh"
#include "nrgpu_fd.cuh"

namespace {

enum { G11 = 0, CHI = 6, A11 = 7, KK = 13, GA1 = 14, ALPHA = 17, BETA1 = 18, BB1 = 21 };
enum { ZG11 = 0, ZCHI = 6, ZA11 = 7, ZKHAT = 13, ZGA1 = 14, ZTHETA = 17, ZALPHA = 18, ZBETA1 = 19, ZBB1 = 22 };
constexpr int ZNV = NRGPU_Z4_NVARS;

// lopsided advection rows (numerators), row r = stencil shifted by r
// (bam_amr_advection.h:28-66); denominators 2, 12, 60
__constant__ double kAdv2[3][3] = {{3, -4, 1}, {1, 0, -1}, {-1, 4, -3}};
__constant__ double kAdv4[5][5] = {{25, -48, 36, -16, 3}, {3, 10, -18, 6, -1}, {-1, 8, 0, -8, 1},
                                   {1, -6, 18, -10, -3}, {-3, 16, -36, 48, -25}};
__constant__ double kAdv6[7][7] = {{147, -360, 450, -400, 225, -72, 10}, {10, 77, -150, 100, -50, 15, -2},
                                   {-2, 24, 35, -80, 30, -8, 1},        {1, -9, 45, 0, -45, 9, -1},
                                   {-1, 8, -30, 80, -35, -24, 2},       {2, -15, 50, -100, 150, -77, -10},
                                   {-10, 72, -225, 400, -450, 360, -147}};

struct AdvDir {
  int base;     // offset of tap 0 relative to the point
  int step;     // +-stride between taps (0 when the shift is zero)
  int row;      // stencil row
};

// direction setup of set_advectionN_onedir (bam_amr_advection.h:72-192)
__device__ __forceinline__ AdvDir adv_dir(int i, int imax, double w, int q, int lop, int s) {
  AdvDir a;
  int rst = q - lop, offset, wsign;
  if (w < 0) { wsign = -1; offset = (i >= rst) ? 0 : rst - i; }
  else if (w > 0) { wsign = 1; offset = (imax - i >= rst) ? 0 : rst - (imax - i); }
  else { wsign = 0; offset = 0; }
  offset += lop;
  a.row = offset;
  a.step = wsign * s;
  a.base = -offset * wsign * s;
  return a;
}

template <int Q>
__device__ __forceinline__ double adv_sum(const double *__restrict__ f, int x, const AdvDir ad[3],
                                          const double cw[3]) {
  double acc = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double t = 0.0;
    const int p0 = x + ad[d].base;
#pragma unroll
    for (int n = 0; n <= Q; ++n) {
      const double c = Q == 2 ? kAdv2[ad[d].row][n] : Q == 4 ? kAdv4[ad[d].row][n] : kAdv6[ad[d].row][n];
      t += c * ldg(f + p0 + n * ad[d].step);
    }
    acc += cw[d] * t;
  }
  return acc;
}

// Kreiss-Oliger: sum over directions of undivided differences / h
template <int OD>
__device__ __forceinline__ double ko_sum(const double *__restrict__ f, int x, const int st[3],
                                         const double ooh[3]) {
  double acc = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int s = st[d];
    double t;
    if (OD == 4)
      t = 6.0 * ldg(f + x) - 4.0 * (ldg(f + x - s) + ldg(f + x + s)) + (ldg(f + x - 2 * s) + ldg(f + x + 2 * s));
    else
      t = (ldg(f + x - 3 * s) + ldg(f + x + 3 * s)) - 6.0 * (ldg(f + x - 2 * s) + ldg(f + x + 2 * s)) +
          15.0 * (ldg(f + x - s) + ldg(f + x + s)) - 20.0 * ldg(f + x);
    acc += ooh[d] * t;
  }
  return OD == 4 ? -acc : acc;
}

// Kreiss-Oliger with FP32 sums of centre-relative taps (the weights sum to
// zero); P = 0 keeps FP64
template <int OD, int P>
__device__ __forceinline__ double ko_p(const double *__restrict__ f, int x, const int st[3], const double ooh[3]) {
  if (P == 0) return ko_sum<OD>(f, x, st, ooh);
  const double c = ldg(f + x);
  double acc = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int s = st[d];
    float t;
    if (OD == 4)
      t = -4.0f * (tapf(f, x, -1, s, c) + tapf(f, x, 1, s, c)) + (tapf(f, x, -2, s, c) + tapf(f, x, 2, s, c));
    else
      t = (tapf(f, x, -3, s, c) + tapf(f, x, 3, s, c)) - 6.0f * (tapf(f, x, -2, s, c) + tapf(f, x, 2, s, c)) +
          15.0f * (tapf(f, x, -1, s, c) + tapf(f, x, 1, s, c));
    acc += ooh[d] * (double)t;
  }
  return OD == 4 ? -acc : acc;
}

struct PointCtx {
  int ijk, i, j, k, imax, jmax, kmax, dist;
  int st[3];
  double h[3];
};

// hints that the line holding p will be read soon: fetched into L1 or L2, no
// register written
__device__ __forceinline__ void l1_prefetch(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
__device__ __forceinline__ void l2_prefetch(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// n: the first 14 variables of either system (g~ at 0..5, A~ at 7..12)
__device__ __forceinline__ void det_trace_fix(double *n, int subtractA, int normalizedetg) {
  double *g = n + G11, *A = n + A11;
  const double detg = g[0] * g[3] * g[5] + 2.0 * g[1] * g[2] * g[4] - g[0] * g[4] * g[4] -
                      g[3] * g[2] * g[2] - g[5] * g[1] * g[1];
  const double detnginv = 1.0 / detg;
  if (subtractA) {
    const double gi0 = g[3] * g[5] - g[4] * g[4], gi1 = g[2] * g[4] - g[1] * g[5],
                 gi2 = g[1] * g[4] - g[2] * g[3], gi3 = g[0] * g[5] - g[2] * g[2],
                 gi4 = g[1] * g[2] - g[0] * g[4], gi5 = g[0] * g[3] - g[1] * g[1];
    const double trA = detnginv * (gi0 * A[0] + gi3 * A[3] + gi5 * A[5] + 2.0 * (gi1 * A[1] + gi2 * A[2] + gi4 * A[4]));
    const double aux = -trA / 3.0;
#pragma unroll
    for (int v = 0; v < 6; ++v) A[v] += aux * g[v];
  }
  if (normalizedetg) {
    const double aux = cbrt(detnginv);
#pragma unroll
    for (int v = 0; v < 6; ++v) g[v] *= aux;
  }
}

}  // namespace
