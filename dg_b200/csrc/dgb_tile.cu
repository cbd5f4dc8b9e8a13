// The tiled 2D residual of structured row-major grids (device/tile2d_cols.cuh): its tables, its
// dispatch over order, flux and field set, and its launches.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstring>
#include <string>
#include <vector>

#include "../../include/dgb.h"
#include "device/kernels.cuh"
#include "device/tile2d_cols.cuh"
#include "device/tile2d_ordered.cuh"
#include "host/host.h"
#include "launch.h"

namespace dgb {

// Tables of the problem with constants cs: for the stage update (M1^-1 and 1/J folded in), or for
// the residual itself (raw: neither).
ColTab make_col_tab(const Consts& cs, bool raw) {
  ColTab t;
  std::memset(&t, 0, sizeof(t));
  const int n1 = cs.n1, ng1 = cs.ng1;
  std::vector<double> M((size_t)n1 * n1, 0.0);  // 1D mass matrix of the reference element, inverted
  for (int i = 0; i < n1; ++i)
    for (int j = 0; j < n1; ++j) {
      if (raw) M[i + (size_t)j * n1] = i == j ? 1.0 : 0.0;
      else
        for (int g = 0; g < ng1; ++g) M[i + (size_t)j * n1] += cs.wq[g] * cs.Bq[g][i] * cs.Bq[g][j];
    }
  if (!raw) invert(M, n1);
  auto fold = [&](const double* row, int i) {
    double s = 0;
    for (int k = 0; k < n1; ++k) s += M[i + (size_t)k * n1] * row[k];
    return s;
  };
  const double jx = raw ? cs.J : 1.0;
  for (int g = 0; g < ng1; ++g)
    for (int i = 0; i < n1; ++i) {
      t.B1[g][i] = cs.Bq[g][i];
      t.Dx[g][i] = cs.ixx * cs.Dq[g][i];
      t.Dy[g][i] = cs.iyy * cs.Dq[g][i];
      t.LB[g][i] = cs.wq[g] * fold(cs.Bq[g], i);
      t.LD[g][i] = cs.wq[g] * fold(cs.Dq[g], i);
      t.XD[g][i] = jx * cs.ixx * cs.wq[g] * fold(cs.Dq[g], i);
      t.XB[g][i] = jx * cs.iyy * cs.wq[g] * fold(cs.Bq[g], i);
      t.XS[g][i] = jx * cs.wq[g] * fold(cs.Bq[g], i);
    }
  for (int g = 0; g < n1; ++g)
    for (int i = 0; i < n1; ++i) {
      t.BF[g][i] = cs.Bf[g][i];
      t.LF[g][i] = 0.5 * cs.wf[g] * fold(cs.Bf[g], i);
    }
  const double fx = raw ? cs.JFx : cs.JFx / cs.J, fy = raw ? cs.JFy : cs.JFy / cs.J;
  for (int i = 0; i < n1; ++i) {
    t.EX[0][i] = fx * M[i];
    t.EX[1][i] = -fx * M[i + (size_t)(n1 - 1) * n1];
    t.EY[0][i] = fy * M[i];
    t.EY[1][i] = -fy * M[i + (size_t)(n1 - 1) * n1];
  }
  return t;
}

namespace {

OrdTab make_ord_tab(const Consts& cs) {
  OrdTab t;
  std::memset(&t, 0, sizeof(t));
  const int n1 = cs.n1, ng1 = cs.ng1;
  std::vector<double> M((size_t)n1 * n1, 0.0);
  for (int i = 0; i < n1; ++i)
    for (int j = 0; j < n1; ++j)
      for (int g = 0; g < ng1; ++g) M[i + (size_t)j * n1] += cs.wq[g] * cs.Bq[g][i] * cs.Bq[g][j];
  invert(M, n1);
  for (int g = 0; g < ng1; ++g) {
    for (int i = 0; i < n1; ++i) { t.B1[g][i] = cs.Bq[g][i]; t.D1[g][i] = cs.Dq[g][i]; }
    for (int h = 0; h < ng1; ++h) t.W[g][h] = cs.wq[g] * cs.wq[h];
  }
  for (int i = 0; i < n1; ++i) {
    t.wf[i] = cs.wf[i];
    for (int j = 0; j < n1; ++j) { t.Bf[i][j] = cs.Bf[i][j]; t.M1i[i][j] = M[i + (size_t)j * n1]; }
  }
  t.cx = cs.J * cs.ixx; t.cy = cs.J * cs.iyy;
  t.sx = cs.ixx; t.sy = cs.iyy;
  t.J = cs.J; t.invJ = 1.0 / cs.J;
  t.JFx = cs.JFx; t.JFy = cs.JFy;
  return t;
}

// The elements in whole 32 x 2 blocks, then the others (all of them on smaller grids) with the generic kernel;
// disjoint outputs, both read the stage input's neighbours from global memory.
template <int FLUX, int MODE, int NY, bool GC>
int launch_ordered(dgb_ctx* c, const StageArgs& s, const ColArgs& a, const CUtensorMap& map, const CUtensorMap& base) {
  if (c->tiled) {
    using Dm = OrdDims<NY, GC>;
    auto k = residual2d_ordered_kernel<FLUX, MODE, NY, GC>;
    DGB_CUDA(allow_dynamic_smem(k, Dm::smem_bytes));
    const int nxt = c->nx / TILE_W * TILE_W, nyt = c->ny / 2 * 2;
    const dim3 grid = tile_grid(nxt / Dm::TW, (nyt + Dm::TH - 1) / Dm::TH);
    ProfScope ps(c, KC_RESIDUAL);
    DGB_CUDA(launch_pdl(c, k, grid, dim3(Dm::NT), Dm::smem_bytes, a, c->ord_tab, nxt, nyt, map, base));
  }
  if (!c->tiled) launch_res2d<3, FLUX, MODE, NY, GC>(c, s);
  else if (c->nleft) launch_res2d<3, FLUX, MODE, NY, GC>(c, s, c->left, c->nleft);
  return 0;
}

template <int NY, bool GC>
int dispatch_ordered(dgb_ctx* c, int mode, const StageArgs& s, const ColArgs& a, const CUtensorMap& map,
                     const CUtensorMap& base) {
  if (c->flux == DGB_FLUX_ROE) {
    return mode == MODE_SSP ? launch_ordered<2, MODE_SSP, NY, GC>(c, s, a, map, base)
                            : launch_ordered<2, MODE_RK4, NY, GC>(c, s, a, map, base);
  }
  return mode == MODE_SSP ? launch_ordered<0, MODE_SSP, NY, GC>(c, s, a, map, base)
                          : launch_ordered<0, MODE_RK4, NY, GC>(c, s, a, map, base);
}

template <int P, int FLUX, int NY, bool GC>
int launch_cols(dgb_ctx* c, const ColArgs& a, const ColTab& tab, const CUtensorMap& map, const CUtensorMap& base) {
  using Dm = ColDims<P, NY, GC>;
  auto k = residual2d_cols_kernel<P, FLUX, NY, GC>;
  DGB_CUDA(allow_dynamic_smem(k, Dm::smem_bytes));
  const dim3 grid = tile_grid((c->nx + Dm::TW - 1) / Dm::TW, (c->ny + Dm::TH - 1) / Dm::TH);
  ProfScope ps(c, KC_RESIDUAL);
  DGB_CUDA(launch_pdl(c, k, grid, dim3(Dm::NT), Dm::smem_bytes, a, tab, map, base));
  return 0;
}

template <int NY, bool GC>
int dispatch_cols(dgb_ctx* c, const ColArgs& a, const ColTab& tab, const CUtensorMap& map, const CUtensorMap& base) {
  switch (c->p * 10 + c->flux) {
    case 10: return launch_cols<1, 0, NY, GC>(c, a, tab, map, base);
    case 12: return launch_cols<1, 2, NY, GC>(c, a, tab, map, base);
    case 20: return launch_cols<2, 0, NY, GC>(c, a, tab, map, base);
    case 22: return launch_cols<2, 2, NY, GC>(c, a, tab, map, base);
    case 30: return launch_cols<3, 0, NY, GC>(c, a, tab, map, base);
    case 32: return launch_cols<3, 2, NY, GC>(c, a, tab, map, base);
    default: return set_error(DGB_ERR_UNSUPPORTED, "no residual kernel for this (dim, p, flux)");
  }
}

}  // namespace

namespace {
template <int P>
void tile_of(const dgb_ctx* c, int& tw, int& th) {
  if (c->gamcons) { tw = ColDims<P, 0, true>::TW; th = ColDims<P, 0, true>::TH; }
  else if (c->nmass > 0) { tw = ColDims<P, 1, false>::TW; th = ColDims<P, 1, false>::TH; }
  else { tw = ColDims<P, 0, false>::TW; th = ColDims<P, 0, false>::TH; }
}
}  // namespace

// Tables and tensor maps of a structured 2D problem.  Rows must start on 16-byte boundaries for TMA (nx
// even) and the grid must hold one tile's box; the other grids take plain loads.
void cols_setup(dgb_ctx* c) {
  c->col_step = make_col_tab(c->cs, false);
  c->col_raw = make_col_tab(c->cs, true);
  if (c->p == 3) c->ord_tab = make_ord_tab(c->cs);
  int tw = 0, th = 0;
  if (c->p == 1) tile_of<1>(c, tw, th);
  else if (c->p == 2) tile_of<2>(c, tw, th);
  else tile_of<3>(c, tw, th);
  c->cols_tma = c->nx % 2 == 0 && c->nx >= tw && c->ny >= th && encode_state_map(c, c->A, &c->colA, tw, th) &&
                encode_state_map(c, c->B, &c->colB, tw, th) && encode_state_map(c, c->C, &c->colC, tw, th) &&
                encode_state_map(c, c->DU, &c->colD, tw, th);
}

int residual2d_cols(dgb_ctx* c, const StageArgs& s, int mode) {
  ColArgs a;
  std::memset(&a, 0, sizeof(a));
  a.U = s.U;
  a.out = s.out;
  a.nbr = s.nbr;
  a.scal = s.scal;
  a.errflag = &c->scal->flags;
  a.polls = c->wait_polls;
  a.nx = c->nx; a.ny = c->ny; a.ld = c->ld;
  a.tma = c->cols_tma ? 1 : 0;
  const ColTab& tab = mode == MODE_RESIDUAL ? c->col_raw : c->col_step;
  a.dt = mode == MODE_RESIDUAL ? 1.0 : s.dt_override;
  if (mode == MODE_SSP) {
    a.base = s.Ubase;
    a.k0 = s.a;
    a.k1 = a.k2 = s.b;
  } else if (s.Us) {  // RK4 with the next stage input: out = Us + beta DU, accumulator = Ubase + b DU
    a.base = s.Us;
    a.k0 = 1.0;
    a.k2 = s.beta_next;
    a.base2 = s.Ubase;
    a.out2 = s.Uacc;
    a.c2 = s.b;
  } else {
    a.k2 = 1.0;
    a.base2 = a.out2 = s.Uacc;
    a.c2 = s.b;
  }
  auto map_of_buf = [&](const double* q) -> const CUtensorMap& {
    return q == c->B ? c->colB : q == c->C ? c->colC : q == c->DU ? c->colD : c->colA;
  };
  const CUtensorMap& map = map_of_buf(s.U);
  const CUtensorMap& base = map_of_buf(a.base);  // read only when k0 != 0
  if (c->ordered() && mode != MODE_RESIDUAL) {
    if (c->gamcons) return dispatch_ordered<0, true>(c, mode, s, a, map, base);
    switch (c->nmass) {
      case 0: return dispatch_ordered<0, false>(c, mode, s, a, map, base);
      case 1: return dispatch_ordered<1, false>(c, mode, s, a, map, base);
      case 2: return dispatch_ordered<2, false>(c, mode, s, a, map, base);
      case 3: return dispatch_ordered<3, false>(c, mode, s, a, map, base);
      default: break;
    }
  }
  if (c->gamcons) return dispatch_cols<0, true>(c, a, tab, map, base);
  switch (c->nmass) {
    case 0: return dispatch_cols<0, false>(c, a, tab, map, base);
    case 1: return dispatch_cols<1, false>(c, a, tab, map, base);
    case 2: return dispatch_cols<2, false>(c, a, tab, map, base);
    case 3: return dispatch_cols<3, false>(c, a, tab, map, base);
    default: return set_error(DGB_ERR_UNSUPPORTED, "no residual kernel for this (dim, p, flux)");
  }
}

}  // namespace dgb
