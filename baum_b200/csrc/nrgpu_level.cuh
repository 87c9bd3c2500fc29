// nrgpu_level.cuh -- device mirror of a BAM level (tL, bam_amr.h:46-74).
#pragma once
#include <mutex>
#include "nrgpu_common.cuh"

// one point with a non-zero boundary flag: linear index, box-local ijk,
// box number and flag; the boundary kernels walk this list
struct FlagPoint {
  int ijk, i, j, k;
  int box, flag;
};

// z slabs of the pipelined host-buffer step (nrgpu_bssn_evolve_host)
#define NRGPU_HOST_SLABS 8

// a symmetry ghost (SYMBOUND point), its mirror image and the reflected
// axes (bit 0 x, 1 y, 2 z): the value is the mirror's times the variable's
// parity under those reflections
struct SymPoint {
  int dst, src, mask;
};

// how an rhs kernel leaves its results
enum { EPI_RHS = 0, EPI_ADDLINEAR = 1, EPI_RK = 2 };

// EPI_RK accumulator modes: ACC_ADD acc += wacc rhs; ACC_INIT acc = upre +
// wacc rhs (the first stage, so that the step needs no copy of u); ACC_FINAL
// out = acc + wacc rhs (the last stage writes u from the accumulator)
enum { ACC_ADD = 0, ACC_INIT = 1, ACC_FINAL = 2 };

struct Epilogue {
  int mode;
  double c;        // EPI_ADDLINEAR: unew = upre + c rhs
  double wacc;     // EPI_RK: acc += wacc * rhs
  double cv;       // EPI_RK: vout = upre + cv * rhs (when has_v)
  int has_v;
  int accmode;     // EPI_RK: ACC_ADD / ACC_INIT / ACC_FINAL
};

// what the interior rhs keeps beside the fields, allocated on first use: the
// lists that the two kernels of nrgpu_deriv.cuh pass from one to the other
// (rows of NRGPU_DERIV_LISTS x NRGPU_DERIV_PITCH doubles), and the staging
// buffer of a box whose size has no compile-time-stride kernel
// (pad_copy_kernel).  Launches that use one of these must not overlap.
struct RhsWork {
  double *lists;
  size_t list_rows;
  int lists_tried;
  double *pad;
  size_t pad_doubles;
  int pad_tried;
};

struct nrgpu_level {
  int device;
  int nboxes;
  int npoints;
  double dx, dy, dz;
  BoxGeo *hbox;            // host copy of the boxes
  int *d_boundary;         // [npoints] flags on the device
  FlagPoint *d_flagpts;    // points with flag != 0
  int nflagpts;
  // flag-0 points within 2 of a box face (the order ladder: lower-order
  // stencils there), sorted by that distance d (FlagPoint.flag = d);
  // nladder[d] = points with distance <= d
  FlagPoint *d_ladder;
  int nladder[3];
  BoxGeo *d_box;           // boxes on the device
  // [0]: NaN flag, [1]: inner point without stencil room, [2], [3]: the queue
  // kernel's tile counters (of the RK steps, of the rhs calls)
  int *d_status;
  // RK4 scratch: three full 24-variable lists, allocated on first use
  double *scratch;
  size_t scratch_points;
  // 1: the interior rhs by the two kernels of nrgpu_deriv.cuh where they
  // cover the run; 0: point by point (nrgpu_level_parts; the levels of a
  // hierarchy of fine spacing, nrgpu_fmr_create)
  int parts;
  // step_work: of the RK steps, which no more overlap each other than they
  // may on the scratch.  call_work: of the rhs calls, which otherwise share
  // nothing and may come from several threads and streams: the lock, and the
  // event of its last use (RhsTurn)
  RhsWork step_work, call_work;
  std::mutex *call_lock;
  cudaEvent_t ev_call;
  // device copy of a host state for the host-buffer entry points
  double *hoststate;
  // points with boundary flag 0, and the norm reduction buffer (first use)
  long ninner;
  double *d_red;
  // partials and results of the 0d output reductions (first use)
  double *d_red0d;
  // extents of the rhs kernels' 128-thread blocks (x, y, z)
  int blk[3];
  // reflection symmetry: the axes (desc.symmetry), the ghost list, and the
  // rhs list of the unfused RK stages of a symmetry grid (first use)
  int symmetry, nsym;
  SymPoint *d_sym;
  double *rsym;
  // side stream of the boundary kernel, which runs beside the interior
  // kernel of the same stage (first use)
  cudaStream_t side;
  cudaEvent_t ev_fork, ev_join;
  // copy and compute streams, and per-slab events, of the pipelined
  // host-buffer step (created on first use)
  cudaStream_t hs_copy, hs_comp;
  cudaEvent_t hev_in[NRGPU_HOST_SLABS], hev_out[NRGPU_HOST_SLABS];
  // interior rhs over TMA-staged tiles (1) instead of per-point global
  // loads (0), where the level and the parameters allow it; the tensor maps
  // of recently used variable lists (host memory, first use)
  int tile;
  // 1: the Z4c interior of all boxes in one persistent launch over a queue
  // of tiles (nrgpu_level_queue), where the boxes allow it
  int queue;
  void *tma_cache;
  int nsm;   // multiprocessors of the level's device
};

// library-internal pieces shared by the entry points and the mesh-refinement
// driver (nrgpu_bssn.cu)
int nrgpu_bssn_rk4_stages(nrgpu_level *L, double *const *u, double dt, const nrgpu_bssn_params *p,
                          cudaStream_t st);
int nrgpu_z4_rk4_stages(nrgpu_level *L, double *const *u, double dt, const nrgpu_z4_params *p, cudaStream_t st);
int nrgpu_z4_algcon(nrgpu_level *L, double *const *u, const nrgpu_z4_params *p, cudaStream_t st);
// set_boundary's background branch for Z4c and the RK4 step that it needs
// (the state's copy kept apart from the extrapolated stage input)
// (nrgpu_z4bg.cu)
int nrgpu_z4_background_extrapolate(nrgpu_level *L, double *const *u, cudaStream_t st);
int nrgpu_z4_background_boundary(nrgpu_level *L, double *const *unew, double *const *upre, double c,
                                 double *const *ucur, const nrgpu_z4_params *p, cudaStream_t st);
// nrgpu_z4_rhs, as a call of its own or inside an RK step
int nrgpu_z4_rhs_of(nrgpu_level *L, bool step, double *const *unew, double *const *upre, double c,
                    double *const *ucur, const nrgpu_z4_params *p, cudaStream_t st);
int nrgpu_z4_rk4_background(nrgpu_level *L, double *const *u, double dt, const nrgpu_z4_params *p, cudaStream_t st);
// the level's three RK4 scratch lists, allocated on first use (nrgpu_lib.cu)
int nrgpu_level_scratch(nrgpu_level *L, double **out);
// the box sizes with a compile-time-stride Z4c rhs kernel; a box of another
// size up to the largest is staged into a copy with the strides of the next
// one (nrgpu_level_reserve)
constexpr int kPadSizes[] = {66, 72, 104, 136, 162, 168, 194};
// the staging size of an m x n box: 0 when it has a kernel of its own or is
// too large
inline int nrgpu_pad_size(int m, int n) {
  if (m == n)
    for (int c : kPadSizes)
      if (c == m) return 0;
  for (int c : kPadSizes)
    if (c >= m && c >= n) return c;
  return 0;
}
// sizes of the lists of the two rhs kernels
#define NRGPU_DERIV_LISTS 71
#define NRGPU_DERIV_PITCH 128
#define NRGPU_PARTS_MIN_POINTS 50000
#define NRGPU_PARTS_MAX_NOISE 4e-14
// what a run's parameters allow on a level: the two kernels (FP64, advection
// rows shifted by 1 or 2 (centred) at 4th order, by 2 or 3 (centred) at 6th; a
// BSSN level whose staged tiles are switched on takes those), and a staging
// copy for the point-by-point kernels
struct RhsRun {
  int order;
  bool two, staged;
};
inline bool nrgpu_two_kernels_rows(int order, int lop, int lop6) {
  return order == 4 ? lop == 1 || lop == 2 : order == 6 && (lop6 == 2 || lop6 == 3);
}
inline RhsRun nrgpu_rhs_run(const nrgpu_level *L, const nrgpu_bssn_params &p) {
  return {p.order_centered,
          L->parts && !L->tile && nrgpu_two_kernels_rows(p.order_centered, p.advection_lopsided, p.advection_lopsided6),
          p.order_centered >= 4};
}
inline RhsRun nrgpu_rhs_run(const nrgpu_level *L, const nrgpu_z4_params &p) {
  return {p.order_centered,
          L->parts && p.precision == 0 &&
              nrgpu_two_kernels_rows(p.order_centered, p.advection_lopsided, p.advection_lopsided6),
          p.order_centered >= 4 && p.precision == 0};
}
// whether a run takes the two kernels on a box, given their lists: the one
// rule of the launches, the allocation and the tuner.  The smallest boxes
// leave most SMs idle either way, and then one launch costs what two do.  Step
// point by point against the two kernels, in us, by inner points (cubes):
//          27000    32768    39304    46656    54872    97336
//   BSSN 4 225/225  380/250  412/245  464/320  475/324  720/510
//   Z4c 4  236/224  404/248  439/270  505/310  522/326  786/536
//   BSSN 6 352/330  582/333  629/381  672/395  758/440
// The line at 50000 is on the safe side of the crossing near 30000, and stays
// there although the boxes between would gain: they have their results to the
// last bit from the point-by-point kernels.
inline bool nrgpu_two_kernels(const RhsRun &run, const BoxGeo &b) {
  const int f = run.order;  // two faces of order / 2 points
  return run.two && b.m > f && b.n > f && b.o > f &&
         (long)(b.m - f) * (b.n - f) * (b.o - f) >= NRGPU_PARTS_MIN_POINTS;
}
// what the run uses of a workspace: the lists, and the staging buffer where a
// box goes point by point; each allocated once, and without memory for them
// the point-by-point kernels run, at run-time strides (nrgpu_lib.cu)
void nrgpu_level_reserve(const nrgpu_level *L, RhsWork *w, const RhsRun &run);
// interior rhs of box b on planes kb .. ke by those kernels, per system and
// order, with the lists of w, where nrgpu_two_kernels holds (nrgpu_parts_*.cu)
void nrgpu_bssn_parts_o4(nrgpu_level *L, const RhsWork &w, int b, const double *const *U, double *const *out,
                         const double *const *pre, double *const *acc, const Epilogue &E, const nrgpu_bssn_params &p,
                         cudaStream_t st, int kb, int ke);
void nrgpu_bssn_parts_o6(nrgpu_level *L, const RhsWork &w, int b, const double *const *U, double *const *out,
                         const double *const *pre, double *const *acc, const Epilogue &E, const nrgpu_bssn_params &p,
                         cudaStream_t st, int kb, int ke);
void nrgpu_z4_parts_o4(nrgpu_level *L, const RhsWork &w, int b, const double *const *U, double *const *out,
                       const double *const *pre, double *const *acc, const Epilogue &E, const nrgpu_z4_params &p,
                       cudaStream_t st, int kb, int ke);
void nrgpu_z4_parts_o6(nrgpu_level *L, const RhsWork &w, int b, const double *const *U, double *const *out,
                       const double *const *pre, double *const *acc, const Epilogue &E, const nrgpu_z4_params &p,
                       cudaStream_t st, int kb, int ke);
// set_boundary_symmetry on a list of nv variables of the given system
// (NRGPU_SYSTEM_BSSN / _Z4C); nothing without symmetry (nrgpu_bssn.cu)
int nrgpu_level_symmetry(nrgpu_level *L, double *const *u, int system, cudaStream_t st);
// the side stream of the boundary kernel (nrgpu_lib.cu)
int nrgpu_level_side(nrgpu_level *L);
// the two halves of a tracking step for a driver that keeps no copy of the
// previous shift: before the step the shift at the old positions into b1,
// after it the corrector passes from b1 (nrgpu_track.cu)
// the extremum search on the given stream (no device switch: graph capture)
int nrgpu_track_extremum_on(nrgpu_level *L, const double *var, int find_max, double minmove, int order, int fixz,
                            int n, double *pos, int *status, cudaStream_t st);
int nrgpu_track_before_step(nrgpu_level *L, const double *const *beta, int order, int n, const double *pos,
                            double *b1, cudaStream_t st);
int nrgpu_track_after_step(nrgpu_level *L, const double *const *beta, double dt, int order, int fixz, int n,
                           double *pos, const double *b1, int *status, cudaStream_t st);
