// nrgpu_deriv.cuh -- the interior right-hand side in two kernels per part of
// a box (included by nrgpu_parts.cuh):
//
//   deriv_kernel    per field: the stencils that several points or several
//                   operators share.  A thread owns one (x, y) column of a
//                   tile and marches along z with the field's planes
//                   k - R .. k + R in registers.  It writes, per point, the
//                   field's advection plus dissipation (weighted, ready to
//                   add to its rhs) and, for the fields that need them, the
//                   numerators d_y f, d_z f and d_zz f.
//   algebra_kernel  per point: d_x f, d_xx f, d_yy f from the field, d_x d_y f,
//                   d_x d_z f and d_y d_z f from the stored numerators of the
//                   columns and rows around (the stencil of
//                   a mixed derivative is the product of two first-derivative
//                   stencils, discretize.m:68-71), then the algebra and the
//                   Runge-Kutta update.
//
// Why: computed point by point from the fields alone, a 4th-order rhs reads
// ~1400 stencil taps per point (a 6th-order one ~2500), most of them for the
// mixed derivatives (16 or 36 each) and for taps that several operators
// share, and it needs every register of the SM for 8 warps that wait for
// those taps.  Here a point costs ~330 loads and ~70 stores in the first
// kernel and ~350 loads in the second, and neither needs compile-time box
// sizes.  The stored numerators lie row by row, all lists of a row side by
// side at a fixed pitch, so that every access to them is one pointer plus a
// constant: with a list per array the address arithmetic was two thirds of
// the instructions that are not FP64.
//
// A part is at most kPartX interior points wide; only d_y f and d_z f are
// needed beyond it, along x, and d_z f along y (H columns and rows on either
// side, which the first kernel computes for both parts).  Along z a part has
// no halo.

// ---- what is stored per row of a part: lists at pitch kPitch ------------------------
//   [0, NV)        advection + dissipation
//   [NV, NV + 3)   advection of Gamma~ alone (only where the B equation takes it)
//   then for the 11 fields with all second derivatives (g~, chi, alpha, beta)
//   d_y, d_z, d_zz, and for the others with first derivatives (Gamma~,
//   K, Theta) d_y, d_z
constexpr int kNM = 11, kPitch = 128, kColumn0 = 4, kPartX = 120;
template <int NV>
struct DerivLists {
  static constexpr int ND = NV == NRGPU_NV ? 4 : 5;
  static constexpr int adv_gamma = NV, dy = NV + 3, dz = dy + kNM, dzz = dz + kNM, ey = dzz + kNM, ez = ey + ND,
                       count = ez + ND;
  // variables: chi 6, K 13, Gamma~ 14, Theta 17 (Z4c), alpha, beta
  static constexpr int alpha = NV == NRGPU_NV ? 17 : 18, beta = alpha + 1;
  // place of variable v among the fields with second, or first, derivatives
  __host__ __device__ static constexpr int im(int v) { return v < 7 ? v : v - alpha + 7; }
  __host__ __device__ static constexpr int id(int v) { return v == 13 ? 3 : v == 17 ? 4 : v - 14; }
};
constexpr int kDerivLists = DerivLists<NRGPU_Z4_NVARS>::count;
static_assert(kDerivLists == NRGPU_DERIV_LISTS && kPitch == NRGPU_DERIV_PITCH, "sizes of the level's lists");

// one part: interior points x0 .. x1, y0 .. y1, z0 .. z1 of the box
struct Part {
  int m, n, o;
  int x0, x1, y0, y1, z0, z1;
};

template <int NV>
struct DerivArgs {
  const double *U[NV];   // fields at the box's first point
  double *ws;
  Part q;
  int chunk, w, tiles_x; // planes per block; tile width and tiles per row of tiles
  int rst, dmin;         // least room for the lopsided rows, least distance for the dissipation
  double ooh[3];
  PartScale<NV> part;    // advection weights times 1 / den1
};

__device__ __forceinline__ double ld(const char *p) { return __ldg((const double *)p); }
__device__ __forceinline__ void st(char *p, double v) { *(double *)p = v; }

// first and second derivative and dissipation numerators from tap differences
// t[r] = f_r - f_-r and sums p[r] = f_r + f_-r, the weights of nrgpu_fd.cuh
template <int ORD>
__device__ __forceinline__ double num1(const double *t) {
  if (ORD == 4) return 8.0 * t[1] - t[2];
  return t[3] - 9.0 * t[2] + 45.0 * t[1];
}
template <int ORD>
__device__ __forceinline__ double num2(const double *p, double c) {
  if (ORD == 4) return 16.0 * p[1] - p[2] - 30.0 * c;
  return 2.0 * p[3] - 27.0 * p[2] + 270.0 * p[1] - 490.0 * c;
}
template <int KOD>
__device__ __forceinline__ double numko(const double *p, double c) {
  if (KOD == 4) return 4.0 * p[1] - p[2] - 6.0 * c;
  return p[3] - 6.0 * p[2] + 15.0 * p[1] - 20.0 * c;
}

// Upwind rows: the lopsided first derivative along +-x is the centred one
// plus an odd and an even high difference,
//   w D_up f = w D1 f + w Q f + |w| S f,
// 4th order shifted by 1: Q = (f_3 - 4 f_2 + 5 f_1 - odd mirror) / 2,
// S = (6th difference) / 2; 6th order shifted by 2: Q = -(f_4 - 6 f_3 +
// 14 f_2 - 14 f_1 - odd mirror) / 2, S = -(8th difference) / 2.  A point
// without room for the lopsided row takes the centred row
// (bam_amr_advection.h:72-192), i.e. drops Q and S.
enum { UP_CENTRED = 0, UP_4 = 1, UP_6 = 2 };

enum { FIELD_PLAIN = 0, FIELD_FIRST = 1, FIELD_SECOND = 2 };

// field v of one column along the planes ka .. kb - 1.  list: where its
// advection + dissipation goes; ko: with dissipation
template <int ORD, int UP, int KOD, int NV, int KIND>
__device__ __forceinline__ void march(const DerivArgs<NV> &a, int v, int list, bool ko, int i, int j, int ka, int kb) {
  using L = DerivLists<NV>;
  constexpr int R = UP == UP_6 ? 4 : 3, H = ORD / 2;  // reach of the taps, of the centred stencils
  constexpr int Q = 2 * R + 2;                        // ring of planes: 2 R + 1 and the next one on its way
  constexpr size_t row = (size_t)L::count * kPitch * sizeof(double);
  const Part &b = a.q;
  const int ys = b.m * 8;
  const size_t plane = (size_t)b.m * b.n * 8;
  const size_t wplane = row * (size_t)(b.y1 - b.y0 + 1 + 2 * H);
  // x taps around the nearest column that has H neighbours: the columns
  // beyond it (only their d_y and d_z are wanted) read in place
  const int xs = (min(max(i, H), b.m - 1 - H) - i) * 8;
  const ptrdiff_t yb = (ptrdiff_t)(min(max(j, H), b.n - 1 - H) - j) * ys;
  const bool xl = i >= R, xh = i < b.m - R, yl = j >= R, yh = j < b.n - R;
  const size_t c0 = i + (size_t)b.m * j;
  const char *F = (const char *)(a.U[v] + c0);
  const double wa = a.part.adv[v], wk = ko ? a.part.ko[v] : 0.0;
  double q[Q];
#pragma unroll
  for (int s = -R; s <= R; ++s) q[s + R] = ld(F + plane * (size_t)min(max(ka + s, 0), b.o - 1));
  F += plane * (size_t)ka;
  char *W = (char *)a.ws + row * (size_t)(j - b.y0 + H) + (size_t)(i - b.x0 + kColumn0) * 8 + wplane * (size_t)(ka - b.z0);
  const char *Bt = (const char *)(a.U[L::beta] + c0) + plane * (size_t)ka;
  const ptrdiff_t b1 = (const char *)a.U[L::beta + 1] - (const char *)a.U[L::beta],
                  b2 = (const char *)a.U[L::beta + 2] - (const char *)a.U[L::beta];
  const int dxy = min(min(i, b.m - 1 - i), min(j, b.n - 1 - j));
  char *M = W + (KIND == FIELD_SECOND ? L::im(v) : L::id(v)) * (kPitch * 8);
  W += list * (kPitch * 8);

  for (int kk = ka; kk < kb; kk += Q) {
#pragma unroll
    for (int s = 0; s < Q; ++s) {
      const int k = kk + s;
      if (k >= kb) return;
      // slot of plane k + r is (s + R + r) mod Q
      const size_t ahead = k + R + 1 < b.o ? plane * (R + 1) : plane * (size_t)(b.o - 1 - k);
      q[(s + 2 * R + 1) % Q] = ld(F + ahead);
      double w[3], wq[3];
      {
        const double bt[3] = {ld(Bt), ld(Bt + b1), ld(Bt + b2)};
        const int at[3] = {i, j, k}, mx[3] = {b.m - 1, b.n - 1, b.o - 1};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          w[d] = bt[d] * a.ooh[d];
          const bool room = (bt[d] < 0.0 ? at[d] : mx[d] - at[d]) >= a.rst;
          wq[d] = room ? (UP == UP_4 ? 0.5 : -0.5) * w[d] : 0.0;
        }
      }
      const bool diss = min(dxy, min(k, b.o - 1 - k)) >= a.dmin;
      const double c = q[(s + R) % Q];
      double adv = 0.0, kos = 0.0, t[R + 1], p[R + 1], ny = 0.0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
#pragma unroll
        for (int r = 1; r <= R; ++r) {
          double lo, hi;
          if (d == 0) {
            lo = r <= H || xl ? ld(F + xs - 8 * r) : c;
            hi = r <= H || xh ? ld(F + xs + 8 * r) : c;
          } else if (d == 1) {
            lo = r <= H || yl ? ld(F + yb - ys * r) : c;
            hi = r <= H || yh ? ld(F + yb + ys * r) : c;
          } else {
            lo = q[(s + R - r + Q) % Q];
            hi = q[(s + R + r) % Q];
          }
          t[r] = hi - lo;
          p[r] = hi + lo;
        }
        const double n1 = num1<ORD>(t), k1 = numko<KOD>(p, c);
        if (d == 1) ny = n1;
        adv += w[d] * n1;
        kos += a.ooh[d] * k1;
        if (UP == UP_4) {
          adv += wq[d] * (t[3] - 4.0 * t[2] + 5.0 * t[1]);
          adv += fabs(wq[d]) * (KOD == 6 ? k1 : numko<6>(p, c));
        }
        if (UP == UP_6) {
          adv += wq[d] * (t[R] - 6.0 * t[3] + 14.0 * t[2] - 14.0 * t[1]);
          adv -= fabs(wq[d]) * (p[R] - 8.0 * p[3] + 28.0 * p[2] - 56.0 * p[1] + 70.0 * c);
        }
      }
      st(W, wa * adv + (diss ? wk * kos : 0.0));
      if (KIND == FIELD_SECOND) {
        st(M + L::dy * (kPitch * 8), ny);
        st(M + L::dz * (kPitch * 8), num1<ORD>(t));
        st(M + L::dzz * (kPitch * 8), num2<ORD>(p, c));
      } else if (KIND == FIELD_FIRST) {
        st(M + L::ey * (kPitch * 8), ny);
        st(M + L::ez * (kPitch * 8), num1<ORD>(t));
      }
      W += wplane;
      Bt += plane;
      M += wplane;
      F += plane;
    }
  }
}

// the fields (blockIdx.z), all of one kind next to each other, so that the
// blocks of an SM run the same code; the last three only where the advection
// of Gamma~ alone is wanted
// 256 threads: a tile of 33 x 7 points reads 13 rows per plane, one of 33 x 3
// (128 threads) 9 for 3, and the L1 misses are those rows (66^3 rhs 213 ->
// 208 us, 136^3 1.93 -> 1.83 ms); three blocks at 80 registers, whose few
// spills cost less than the warps of a third block gain
constexpr int kDerivThreads = 256;

template <int ORD, int UP, int KOD, int NV>
__global__ void __launch_bounds__(kDerivThreads, UP == UP_6 ? 2 : 3) deriv_kernel(const DerivArgs<NV> a) {
  using L = DerivLists<NV>;
  constexpr int H = ORD / 2;
  const int tx = blockIdx.x % a.tiles_x, ty = blockIdx.x / a.tiles_x;
  const int rows = kDerivThreads / a.w, lj = threadIdx.x / a.w;
  const int i = a.q.x0 - H + tx * a.w + threadIdx.x - lj * a.w, j = a.q.y0 - H + ty * rows + lj;
  if (lj >= rows || i > a.q.x1 + H || j > a.q.y1 + H) return;
  const int ka = a.q.z0 + blockIdx.y * a.chunk, kb = min(ka + a.chunk, a.q.z1 + 1);
  int g = blockIdx.z;
  if (g < kNM) {
    const int v = g < 7 ? g : L::alpha + g - 7;
    march<ORD, UP, KOD, NV, FIELD_SECOND>(a, v, v, true, i, j, ka, kb);
  } else if ((g -= kNM) < L::ND) {
    const int v = g == 4 ? 17 : 13 + g;
    march<ORD, UP, KOD, NV, FIELD_FIRST>(a, v, v, true, i, j, ka, kb);
  } else {
    // A~, B, then the advection of Gamma~
    g -= L::ND;
    const int v = g < 6 ? 7 + g : g < 9 ? L::beta + g - 3 : 14 + g - 9;
    march<ORD, UP, KOD, NV, FIELD_PLAIN>(a, v, g < 9 ? v : L::adv_gamma + g - 9, g < 9, i, j, ka, kb);
  }
}

// ---- the algebra kernel ------------------------------------------------------------
template <int ORD, int NV>
struct PartSource {
  using L = DerivLists<NV>;
  const double *const *U;  // fields at the box's first point
  size_t x;                // the point, in the fields
  const char *W;           // the point, in the first list
  int ys;                  // bytes of a row of the fields

  __device__ __forceinline__ const char *field(int v) const { return (const char *)(U[v] + x); }
  __device__ __forceinline__ double val(int v) const { return ld(field(v)); }
  __device__ __forceinline__ double list(int q, int r = 0) const { return ld(W + q * kPitch * 8 + 8 * r); }
  // d_x of a list
  __device__ __forceinline__ double dx_list(int q) const {
    double t[4];
#pragma unroll
    for (int r = 1; r <= ORD / 2; ++r) t[r] = list(q, r) - list(q, -r);
    return num1<ORD>(t);
  }
  __device__ __forceinline__ void d1(int v, double n1[3]) const {
    double t[4];
    const char *F = field(v);
#pragma unroll
    for (int r = 1; r <= ORD / 2; ++r) t[r] = ld(F + 8 * r) - ld(F - 8 * r);
    n1[0] = num1<ORD>(t);
    n1[1] = list(L::ey + L::id(v));
    n1[2] = list(L::ez + L::id(v));
  }
  __device__ __forceinline__ void jet(int v, double n1[3], double n2[6]) const {
    const char *F = field(v);
    double t[4], p[4];
    const double c = ld(F);
#pragma unroll
    for (int r = 1; r <= ORD / 2; ++r) {
      const double hi = ld(F + 8 * r), lo = ld(F - 8 * r);
      t[r] = hi - lo;
      p[r] = hi + lo;
    }
    n1[0] = num1<ORD>(t);
    n2[0] = num2<ORD>(p, c);
#pragma unroll
    for (int r = 1; r <= ORD / 2; ++r) p[r] = ld(F + ys * r) + ld(F - ys * r);
    n2[3] = num2<ORD>(p, c);
    n1[1] = list(L::dy + L::im(v));
    n1[2] = list(L::dz + L::im(v));
    n2[1] = dx_list(L::dy + L::im(v));
    n2[2] = dx_list(L::dz + L::im(v));
    {
      // d_y of d_z f: the rows of a plane lie one after another
      double t[4];
#pragma unroll
      for (int r = 1; r <= ORD / 2; ++r) t[r] = list(L::dz + L::im(v) + L::count * r) - list(L::dz + L::im(v) - L::count * r);
      n2[4] = num1<ORD>(t);
    }
    n2[5] = list(L::dzz + L::im(v));
  }
  __device__ __forceinline__ double add_part(int v, double r) const { return r + list(v); }
  __device__ __forceinline__ double adv_gamma(int a) const { return list(L::adv_gamma + a); }
};

// where the results of a point go.  EPI_RHS: dst1 = r.  EPI_RK: dst1 = base +
// w1 r and, with has2, dst2 = pre + w2 r (first stage: base = pre, dst1 the
// accumulator; middle stages: base = dst1 = the accumulator; last stage:
// base the accumulator, dst1 the state).  EPI_ADDLINEAR: dst1 = base + w1 r
// with the determinant and trace fixed.
template <int NV>
struct SinkArgs {
  double *dst1[NV], *dst2[NV];
  const double *base[NV], *pre[NV];
  double w1, w2;
  int has2;
};

template <int NV, int MODE>
struct PartSink {
  const SinkArgs<NV> &a;
  size_t x;
  double sum;
  double n[MODE == EPI_ADDLINEAR ? 14 : 1];

  template <int N>
  __device__ __forceinline__ void put(int v, const double *r) {
#pragma unroll
    for (int q = 0; q < N; ++q) sum += r[q];
    if (MODE == EPI_RHS) {
#pragma unroll
      for (int q = 0; q < N; ++q) a.dst1[v + q][x] = r[q];
    } else if (MODE == EPI_RK) {
      double b[N], u[N];
#pragma unroll
      for (int q = 0; q < N; ++q) {
        b[q] = a.base[v + q][x];
        u[q] = a.has2 ? ldg(a.pre[v + q] + x) : 0.0;
      }
#pragma unroll
      for (int q = 0; q < N; ++q) {
        a.dst1[v + q][x] = b[q] + a.w1 * r[q];
        if (a.has2) a.dst2[v + q][x] = u[q] + a.w2 * r[q];
      }
    } else {
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const double y = a.base[v + q][x] + a.w1 * r[q];
        if (v + q < 14) n[v + q < 14 ? v + q : 0] = y;
        else a.dst1[v + q][x] = y;
      }
    }
  }
};

struct AlgebraGeo {
  const double *ws;
  const int *flag;  // boundary flags at the box's first point
  Part q;
  int w, tiles_x;   // tile width and tiles per row of tiles
  DerivScale c;
};

// two blocks of 128 at 254 registers (168 registers and three blocks: spills,
// 3.0 -> 3.3 ms per 162^3 rhs)
constexpr int kAlgebraThreads = 128;

template <int ORD, int NV, int MODE, class PARAMS>
__global__ void __launch_bounds__(kAlgebraThreads, 2)
    algebra_kernel(const CPtrs<NV> U, const AlgebraGeo g, const SinkArgs<NV> sa, const PARAMS p, int *status) {
  using L = DerivLists<NV>;
  const Part &b = g.q;
  const int tx = blockIdx.x % g.tiles_x, ty = blockIdx.x / g.tiles_x;
  const int rows = kAlgebraThreads / g.w, lj = threadIdx.x / g.w;
  const int i = b.x0 + tx * g.w + threadIdx.x - lj * g.w, j = b.y0 + ty * rows + lj, k = b.z0 + blockIdx.y;
  if (lj >= rows || i > b.x1 || j > b.y1) return;
  const size_t x = (size_t)b.m * ((size_t)b.n * k + j) + i;
  if (__ldg(g.flag + x) != 0) return;
  const char *W = (const char *)g.ws +
                  8 * (((size_t)(k - b.z0) * (b.y1 - b.y0 + 1 + ORD) + (j - b.y0 + ORD / 2)) * (L::count * kPitch) +
                       (i - b.x0 + kColumn0));
  // everything of this point that no register has to wait for: the lists and
  // the fields into L1, the update's operands into L2 (66^3 step 1054 ->
  // 999 us, 136^3 10.8 -> 9.6 ms: what the kernel waits for is the latency of
  // its loads, at 8 warps per SM and a register per load in flight)
#pragma unroll
  for (int q = 0; q < L::count; ++q)
    if (q < L::adv_gamma || q >= L::dy) l1_prefetch(W + q * kPitch * 8);
#pragma unroll
  for (int v = 0; v < NV; ++v) l1_prefetch(U.p[v] + x);
  if (MODE == EPI_RK) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      l2_prefetch(sa.base[v] + x);
      if (sa.has2) l2_prefetch(sa.pre[v] + x);
    }
  }
  const PartSource<ORD, NV> s = {U.p, x, W, b.m * 8};
  PartSink<NV, MODE> e = {sa, x, 0.0};
  if constexpr (NV == NRGPU_NV) bssn_algebra(s, g.c, p, e);
  else z4_algebra(s, g.c, p, e);
  if (!isfinite(e.sum)) atomicOr(status, 1);
  if (MODE == EPI_ADDLINEAR) {
    if constexpr (NV == NRGPU_NV) e.n[KK] *= p.forceKzerofactor;
    det_trace_fix(e.n, p.subtractA, p.normalizedetg);
#pragma unroll
    for (int v = 0; v < 14; ++v) sa.dst1[v][x] = e.n[v];
  }
}
