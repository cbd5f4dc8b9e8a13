// Residual + stage update of cubic elements under a limiter on structured grids, with the terms of
// every sum, their order and their rounding fixed.
//
// Why: the limited scheme at p = 3 multiplies rounding differences by 10 to 15 per step (see HrTab3,
// common.cuh), so a run repeats earlier results only if its arithmetic does.  cols_body
// (tile2d_cols.cuh) folds M^-1, weights and metric into its tables and lifts faces before it adds them;
// here every factor is applied on its own, in this order:
//   point values   x contraction, then y, ascending nodes from 0
//   residual node  from 0: left, right, bottom, top face, ascending face points; then the quadrature
//                  columns gx ascending, each l'(x) Ax + l(x) Ay (alpha: l(x) As)
//   update         M1^-1 along x, then along y, times dt / J
//   fluxes         phys::riemann2d_rcp and point_terms with correctly rounded reciprocals and roots
// It covers the elements in whole 32 x 2 blocks; those to the right and above keep the generic kernel
// (residual2d_kernel), whose sums are other ones.
//
// The work is split as in cols_body: a thread per (element, quadrature column), per face point, per
// (element, field, y-node); the unlifted face fluxes, the column sums and the x half of M^-1 pass through
// shared memory.  Per launch at 1024 x 512, Roe: 568 us (RK4, with the accumulator: 690).  One thread per element
// with all its sums in registers and the next RK4 input formed by a kernel of its own took 906 (1,690), and
// cols_body, with its 15 % fewer operations and one shared-memory pass less, takes 421.
#pragma once
#include "kernels.cuh"
#include "tile2d.cuh"
#include "tile2d_cols.cuh"

namespace dgb {

// 1D factors of the reference element (p = 3), by value: constant-bank operands
struct OrdTab {
  double B1[MAXG][MAXN], D1[MAXG][MAXN];  // l_i(x_g), l_i'(x_g)
  double W[MAXG][MAXG];                   // w_gx w_gy
  double Bf[MAXN][MAXN], wf[MAXN];        // l_j on the face's Gauss points, their weights
  double M1i[MAXN][MAXN];                 // inverse of the 1D mass matrix
  double cx, cy, sx, sy, J, invJ, JFx, JFy;  // metric (as in TileArgs)
};

template <int NY, bool GC>
struct OrdDims : ColDims<3, NY, GC> {
  using B = ColDims<3, NY, GC>;
  static constexpr size_t off_half = B::smem_bytes;  // [NF*NS][NE] x half of M^-1
  static constexpr size_t smem_bytes = off_half + B::tile_bytes;
  static constexpr int by_smem = (int)(227 * 1024 / (smem_bytes + 1024));
  static constexpr int ctas = by_smem < 1 ? 1 : by_smem < B::by_regs ? by_smem : B::by_regs < 1 ? 1 : B::by_regs;
};

// nxt, nyt: extents of the covered elements.  MODE_SSP: out = k0 base + k1 (U + du); MODE_RK4: out = base + k2 du
// (k0 == 0: no base, nor is it read), out2 = base2 + c2 du.
template <int FLUX, int MODE, int NY, bool GC>
__global__ void __launch_bounds__(OrdDims<NY, GC>::NT, OrdDims<NY, GC>::ctas)
    residual2d_ordered_kernel(const __grid_constant__ ColArgs a, const __grid_constant__ OrdTab tab, int nxt, int nyt,
                              const __grid_constant__ CUtensorMap mapU, const __grid_constant__ CUtensorMap mapBase) {
  using Dm = OrdDims<NY, GC>;
  constexpr int P = 3, N1 = 4, NS = 16, NF = Dm::NF, NFL = Dm::NFL, NG1 = Dm::NG1, NE = Dm::NE, NT = Dm::NT;
  constexpr int TW = Dm::TW, TH = Dm::TH, NXF = Dm::NXF, NFACE = Dm::NFACE, NEDGE = Dm::NEDGE;
  extern __shared__ __align__(128) unsigned char smraw[];
  int* codes = reinterpret_cast<int*>(smraw + Dm::off_code);
  double* Us = reinterpret_cast<double*>(smraw + Dm::off_tile);    // [NF*NS][NE]
  double* HS = reinterpret_cast<double*>(smraw + Dm::off_halo);    // [NF*N1][NEDGE]
  double* FS = reinterpret_cast<double*>(smraw + Dm::off_face);    // [(NF+1)*N1][NFACE] fluxes, ncterm
  double* AS = reinterpret_cast<double*>(smraw + Dm::off_sums);    // [NA][NT]
  double* HM = reinterpret_cast<double*>(smraw + Dm::off_half);
  if (threadIdx.x == 0) {
    mbar_init(reinterpret_cast<uint64_t*>(smraw), 1);
    fence_mbar_init();
  }
  pdl_wait();
  uint32_t phase = 0;
  const int tid = threadIdx.x, tx0 = blockIdx.x * TW, ty0 = tile_row() * TH;
  if (ty0 >= nyt) return;
  const int tw = min(TW, nxt - tx0), th = min(TH, nyt - ty0);
  if (!cols_load<Dm, P>(a, &mapU, &mapBase, tx0, ty0, tw, th, smraw, phase)) return;

  // ---------------- volume: one thread per (element, quadrature column) ----------------
  {
    const int el = tid % NE, gx = tid / NE;
    if (el / TW < th) {
      double Tc[NF][N1], dT[N1];
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) {
#pragma unroll
        for (int f = 0; f < NF; ++f) {
          double s = 0;
#pragma unroll
          for (int ix = 0; ix < N1; ++ix) s += tab.B1[gx][ix] * Us[(f * NS + ix + N1 * iy) * NE + el];
          Tc[f][iy] = s;
        }
        double sd = 0;
#pragma unroll
        for (int ix = 0; ix < N1; ++ix) sd += tab.D1[gx][ix] * Us[(4 * NS + ix + N1 * iy) * NE + el];
        dT[iy] = sd;
      }
      double Ax[NFL][N1], Ay[NFL][N1], As[N1];
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) {
        As[iy] = 0.0;
#pragma unroll
        for (int f = 0; f < NFL; ++f) Ax[f][iy] = Ay[f][iy] = 0.0;
      }
#pragma unroll
      for (int gy = 0; gy < NG1; ++gy) {
        double ug[NF], dax = 0, day = 0;
#pragma unroll
        for (int f = 0; f < NF; ++f) {
          double s = 0;
#pragma unroll
          for (int iy = 0; iy < N1; ++iy) s += tab.B1[gy][iy] * Tc[f][iy];
          ug[f] = s;
        }
#pragma unroll
        for (int iy = 0; iy < N1; ++iy) { dax += tab.B1[gy][iy] * dT[iy]; day += tab.D1[gy][iy] * Tc[4][iy]; }
        double gxv[NFL], gyv[NFL], gs;
        point_terms<NF, NFL, NY, GC, true>(ug, dax, day, tab.W[gx][gy], tab, gxv, gyv, gs);
#pragma unroll
        for (int iy = 0; iy < N1; ++iy) {
          const double b = tab.B1[gy][iy], d = tab.D1[gy][iy];
#pragma unroll
          for (int f = 0; f < NFL; ++f) { Ax[f][iy] += b * gxv[f]; Ay[f][iy] += d * gyv[f]; }
          if (!GC) As[iy] += b * gs;
        }
      }
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) {
#pragma unroll
        for (int f = 0; f < NFL; ++f) {
          AS[(f * N1 + iy) * NT + tid] = Ax[f][iy];
          AS[((NFL + f) * N1 + iy) * NT + tid] = Ay[f][iy];
        }
        if (!GC) AS[(2 * NFL * N1 + iy) * NT + tid] = As[iy];
      }
    }
  }

  // ---------------- faces: one thread per face point; the left / bottom element is L ----------------
  // (boundary faces: the inside element is L with its outward normal; those seen from the right / top element store
  // -F, so that left and bottom faces give +F + nc and right and top faces -F + nc)
  for (int k = tid; k < N1 * NFACE; k += NT) {
    const int g = k / NFACE, fc = k % NFACE;
    const bool xf = fc < NXF;
    const int kk = xf ? fc : fc - NXF;
    const int fx = xf ? kk % (TW + 1) : kk % TW, fy = xf ? kk / (TW + 1) : kk / TW;
    if (xf ? fy >= th : fy > th) continue;
    const int pos = xf ? fx : fy, last = xf ? TW : th;
    const int slot = xf ? (pos == 0 ? fy : TH + fy) : 2 * TH + (pos == 0 ? 0 : TW) + fx;
    const int code = pos == 0 || pos == last ? codes[slot] : 0;
    const int elR = fy * TW + fx, elL = xf ? elR - 1 : elR - TW, sj = xf ? N1 * NE : NE;
    const double* pL = Us + (xf ? P : N1 * P) * NE + elL;
    const double* pR = Us + elR;
    int sfL = NS * NE, sjL = sj, sfR = NS * NE, sjR = sj;
    if (pos == 0) { pL = HS + slot; sfL = N1 * NEDGE; sjL = NEDGE; }
    else if (pos == last) { pR = HS + slot; sfR = N1 * NEDGE; sjR = NEDGE; }
    double nxv = xf ? 1.0 : 0.0, nyv = xf ? 0.0 : 1.0, sgn = 1.0;
    if (code < 0) {
      if (pos == 0) { pL = pR; sfL = sfR; sjL = sjR; nxv = -nxv; nyv = -nyv; sgn = -1.0; }
      else { pR = pL; sfR = sfL; sjR = sjL; }
    }
    const int mom = code == -3 ? (xf ? 1 : 2) : -1;  // the mirrored momentum (boundaries.cu:20-67)
    double L[NF], R[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      double sl = 0, sr = 0;
#pragma unroll
      for (int j = 0; j < N1; ++j) {
        const double vr = pR[f * sfR + j * sjR];
        sl += tab.Bf[g][j] * pL[f * sfL + j * sjL];
        sr += tab.Bf[g][j] * (f == mom ? -vr : vr);
      }
      L[f] = sl;
      R[f] = sr;
    }
    double F[NF], nc;
    phys::riemann2d_rcp<FLUX, NY, GC, true>(L, R, nxv, nyv, F, nc);
#pragma unroll
    for (int f = 0; f < NF; ++f) FS[(f * N1 + g) * NFACE + fc] = sgn * F[f];
    FS[(NF * N1 + g) * NFACE + fc] = nc;
  }

  // ---------------- update: one thread per (element, field, y-node) ----------------
  constexpr int NIT = (NF * N1 + NG1 - 1) / NG1;
  const unsigned plane = a.ld;
  const int el = tid % NE, tx = el % TW, ty = el / TW, r0 = tid / NE;
  const bool own = ty < th;
  const unsigned g0 = N1 * r0 * plane + (unsigned)((ty0 + ty) * a.nx + tx0 + tx);
  const bool two = MODE == MODE_RK4 && a.out2;
  const double *base = after_wait(a.base), *base2 = after_wait(a.base2);
  double v0[NIT][N1], v2[NIT][N1];
#pragma unroll
  for (int q = 0; q < NIT; ++q) {
    const bool on = own && r0 + q * NG1 < NF * N1;
#pragma unroll
    for (int ix = 0; ix < N1; ++ix) {
      const unsigned gi = g0 + (q * NG1 * N1 + ix) * plane;
      v0[q][ix] = on && a.k0 != 0.0 ? ld_after(base + gi) : 0.0;
      v2[q][ix] = on && two ? ld_after(base2 + gi) : 0.0;
    }
  }
  const double dt = a.dt > 0 ? a.dt : ld_dep(&a.scal->dt);
  const double sc = dt * tab.invJ;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NIT; ++q) {
    const int r = r0 + q * NG1, f = r / N1, iy = r % N1;
    if (!own || r >= NF * N1) break;
    const bool alpha = f == 4;
    double rr[N1] = {0.0, 0.0, 0.0, 0.0};
    const double* fp = FS + f * N1 * NFACE;
    const double* np = FS + NF * N1 * NFACE;
    const int xl = ty * (TW + 1) + tx, yd = NXF + el;
    // +F + nc on the left and bottom faces, -F + nc on the right and top ones
    auto plus = [&](int g, int fc) { return fp[g * NFACE + fc] + (alpha ? np[g * NFACE + fc] : 0.0); };
    auto minus = [&](int g, int fc) { return -fp[g * NFACE + fc] + (alpha ? np[g * NFACE + fc] : 0.0); };
#pragma unroll
    for (int g = 0; g < N1; ++g) rr[0] += tab.Bf[g][iy] * (plus(g, xl) * (tab.JFx * tab.wf[g]));
#pragma unroll
    for (int g = 0; g < N1; ++g) rr[P] += tab.Bf[g][iy] * (minus(g, xl + 1) * (tab.JFx * tab.wf[g]));
    if (iy == 0) {
#pragma unroll
      for (int g = 0; g < N1; ++g) {
        const double c = plus(g, yd) * (tab.JFy * tab.wf[g]);
#pragma unroll
        for (int ix = 0; ix < N1; ++ix) rr[ix] += tab.Bf[g][ix] * c;
      }
    }
    if (iy == P) {
#pragma unroll
      for (int g = 0; g < N1; ++g) {
        const double c = minus(g, yd + TW) * (tab.JFy * tab.wf[g]);
#pragma unroll
        for (int ix = 0; ix < N1; ++ix) rr[ix] += tab.Bf[g][ix] * c;
      }
    }
    if (!GC && alpha) {
      const double* as = AS + (2 * NFL * N1 + iy) * NT + el;
#pragma unroll
      for (int gx = 0; gx < NG1; ++gx) {
        const double v = as[gx * NE];
#pragma unroll
        for (int ix = 0; ix < N1; ++ix) rr[ix] += tab.B1[gx][ix] * v;
      }
    } else {
      const double* as = AS + (GC || r < 4 * N1 ? r : r - N1) * NT + el;
#pragma unroll
      for (int gx = 0; gx < NG1; ++gx) {
        const double vx = as[gx * NE], vy = as[NFL * N1 * NT + gx * NE];
#pragma unroll
        for (int ix = 0; ix < N1; ++ix) rr[ix] += tab.D1[gx][ix] * vx + tab.B1[gx][ix] * vy;
      }
    }
#pragma unroll
    for (int ix = 0; ix < N1; ++ix) {
      double s = 0;
#pragma unroll
      for (int k = 0; k < N1; ++k) s += tab.M1i[ix][k] * rr[k];
      HM[(N1 * r + ix) * NE + el] = s;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NIT; ++q) {
    const int r = r0 + q * NG1, iy = r % N1;
    if (!own || r >= NF * N1) break;
    const double* hm = HM + N1 * (r - iy) * NE + el;
#pragma unroll
    for (int ix = 0; ix < N1; ++ix) {
      double s = 0;
#pragma unroll
      for (int k = 0; k < N1; ++k) s += tab.M1i[iy][k] * hm[(ix + N1 * k) * NE];
      const double du = __dmul_rn(sc, s);
      const unsigned gi = g0 + (q * NG1 * N1 + ix) * plane;
      if (MODE == MODE_SSP) {
        // one rounding for U + du, two for the last value of the element
        const double us = Us[(N1 * r + ix) * NE + el];
        const double t = N1 * r + ix == NF * NS - 1 ? __dadd_rn(us, du) : __fma_rn(sc, s, us);
        a.out[gi] = __fma_rn(a.k1, t, a.k0 != 0.0 ? __dmul_rn(a.k0, v0[q][ix]) : 0.0);
      } else {
        a.out[gi] = v0[q][ix] + a.k2 * du;
        if (two) a.out2[gi] = v2[q][ix] + a.c2 * du;
      }
    }
  }
  pdl_trigger();
}

}  // namespace dgb
