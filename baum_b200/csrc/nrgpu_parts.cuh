// nrgpu_parts.cuh -- host side of the two rhs kernels of nrgpu_deriv.cuh: the
// parts of a box, their tiles and launches.  One translation unit per system
// and order (nrgpu_parts_*.cu).
#pragma once
#include <algorithm>
#include "nrgpu_rhs.cuh"

namespace {

#include "nrgpu_algebra.cuh"
#include "nrgpu_deriv.cuh"

// ---- the two kernels of one box ------------------------------------------------
// tile width of a kernel whose blocks of `threads` cover w x (threads / w)
// points of an nx x ny plane: the one that leaves the fewest threads idle,
// equal widths of 28 to 64 (a warp's access to a row of 28 to 32 points is
// two or three 128-byte lines, to shorter rows one more for each row)
int tile_width(int nx, int ny, int threads) {
  int best = nx < 32 ? nx : 32;
  double eff = 0.0;
  for (int nt = (nx + 63) / 64; nt == 1 || nx / nt >= 28; ++nt) {
    const int w = (nx + nt - 1) / nt, rows = threads / w;
    if (rows < 1) continue;
    const double e = (double)nx * ny / ((double)((nx + w - 1) / w) * ((ny + rows - 1) / rows) * threads);
    if (e > eff + 1e-3) {
      eff = e;
      best = w;
    }
  }
  return best;
}

template <int NV, int ORD, int UP, int KOD>
void launch_deriv(const DerivArgs<NV> &a, bool adv_gamma, cudaStream_t st) {
  const Part &q = a.q;
  const int rows = kDerivThreads / a.w;
  const dim3 grd(a.tiles_x * ((q.y1 - q.y0 + ORD + rows) / rows), (q.z1 - q.z0 + a.chunk) / a.chunk,
                 NV + (adv_gamma ? 3 : 0));
  deriv_kernel<ORD, UP, KOD, NV><<<grd, kDerivThreads, 0, st>>>(a);
}

template <int NV, int ORD, class PARAMS>
void launch_algebra(const CPtrs<NV> &U, const AlgebraGeo &g, const SinkArgs<NV> &sa, const PARAMS &p, int mode,
                           int *status, cudaStream_t st) {
  const Part &q = g.q;
  const int rows = kAlgebraThreads / g.w;
  const dim3 grd(g.tiles_x * ((q.y1 - q.y0 + rows) / rows), q.z1 - q.z0 + 1);
  if (mode == EPI_RK) algebra_kernel<ORD, NV, EPI_RK><<<grd, kAlgebraThreads, 0, st>>>(U, g, sa, p, status);
  else if (mode == EPI_RHS) algebra_kernel<ORD, NV, EPI_RHS><<<grd, kAlgebraThreads, 0, st>>>(U, g, sa, p, status);
  else algebra_kernel<ORD, NV, EPI_ADDLINEAR><<<grd, kAlgebraThreads, 0, st>>>(U, g, sa, p, status);
}

// n points cut into the fewest equal parts of at most `most`
int part_size(int n, int most) {
  const int parts = (n + most - 1) / most;
  return (n + parts - 1) / parts;
}

// interior rhs of box b on planes kb .. ke by the two kernels of
// nrgpu_deriv.cuh, part by part
template <int NV, int ORD, class PARAMS>
void launch_parts(nrgpu_level *L, const RhsWork &w, int b, const double *const *U, double *const *out,
                  const double *const *pre, double *const *acc, const Epilogue &E, const PARAMS &p, cudaStream_t st,
                  int kb, int ke) {
  constexpr int H = ORD / 2;
  const int lop = ORD == 4 ? p.advection_lopsided : p.advection_lopsided6;
  const BoxGeo &bx = L->hbox[b];
  const int z0 = std::max(kb, H), z1 = std::min(ke, bx.o - 1 - H);
  const int nx = bx.m - 2 * H, ny = bx.n - 2 * H, nz = z1 - z0 + 1;
  if (nz < 1) return;  // ladder points only
  const size_t rows = w.list_rows;
  const int px = part_size(nx, kPartX);
  const int py = part_size(ny, (int)std::min<size_t>(rows - 2 * H, ny));
  const int pz = part_size(nz, (int)std::min<size_t>(rows / (py + 2 * H), nz));
  DerivArgs<NV> d;
  AlgebraGeo g;
  CPtrs<NV> cu;
  SinkArgs<NV> sa;
  const bool last = E.mode == EPI_RK && E.accmode == ACC_FINAL;
  for (int v = 0; v < NV; ++v) {
    d.U[v] = cu.p[v] = U[v] + bx.noffset;
    sa.pre[v] = pre[v] + bx.noffset;
    sa.dst2[v] = out[v] + bx.noffset;
    sa.dst1[v] = (E.mode == EPI_RK && !last ? acc[v] : out[v]) + bx.noffset;
    sa.base[v] = (E.mode == EPI_RK && E.accmode != ACC_INIT ? acc[v] : pre[v]) + bx.noffset;
  }
  sa.w1 = E.mode == EPI_RK ? E.wacc : E.c;
  sa.w2 = E.cv;
  sa.has2 = E.mode == EPI_RK && !last && E.has_v;
  g.c = deriv_scale(ORD, L->dx, L->dy, L->dz);
  g.ws = d.ws = w.lists;
  g.flag = L->d_boundary + bx.noffset;
  d.rst = ORD - lop;
  d.dmin = p.order_dissipation == 4 ? 2 : 3;
  d.part = part_scale(p);
  for (int v = 0; v < NV; ++v) d.part.adv[v] *= ORD == 4 ? 1.0 / 12.0 : 1.0 / 60.0;
  for (int a = 0; a < 3; ++a) d.ooh[a] = g.c.ooh[a];
  const bool ko4 = p.order_dissipation == 4, ag = p.withGadv != 1.0, up = lop != ORD / 2;
  constexpr int UP = ORD == 4 ? UP_4 : UP_6;
  Part &q = d.q;
  q.m = bx.m;
  q.n = bx.n;
  q.o = bx.o;
  for (q.z0 = z0; q.z0 <= z1; q.z0 += pz)
    for (q.y0 = H; q.y0 < H + ny; q.y0 += py)
      for (q.x0 = H; q.x0 < H + nx; q.x0 += px) {
        q.z1 = std::min(q.z0 + pz - 1, z1);
        q.y1 = std::min(q.y0 + py, H + ny) - 1;
        q.x1 = std::min(q.x0 + px, H + nx) - 1;
        const int wx = q.x1 - q.x0 + 1, wy = q.y1 - q.y0 + 1, wz = q.z1 - q.z0 + 1;
        d.w = tile_width(wx + 2 * H, wy + 2 * H, kDerivThreads);
        d.tiles_x = (wx + 2 * H + d.w - 1) / d.w;
        const int dr = kDerivThreads / d.w;
        const long tiles = (long)d.tiles_x * ((wy + 2 * H + dr - 1) / dr) * NV;
        // planes per block: enough blocks for every SM, each long enough to
        // pay for the planes a march reads before its first
        int chunks = 1;
        while (wz / (chunks + 1) >= 8 && tiles * chunks < 8L * L->nsm) ++chunks;
        d.chunk = (wz + chunks - 1) / chunks;
        if (up) ko4 ? launch_deriv<NV, ORD, UP, 4>(d, ag, st) : launch_deriv<NV, ORD, UP, 6>(d, ag, st);
        else ko4 ? launch_deriv<NV, ORD, UP_CENTRED, 4>(d, ag, st) : launch_deriv<NV, ORD, UP_CENTRED, 6>(d, ag, st);
        g.q = q;
        g.w = tile_width(wx, wy, kAlgebraThreads);
        g.tiles_x = (wx + g.w - 1) / g.w;
        launch_algebra<NV, ORD>(cu, g, sa, p, E.mode, L->d_status, st);
      }
}

}  // namespace
