// Tiled 2D residual + stage update for structured (row-major nx x ny) Cartesian meshes, one thread
// per (element, quadrature column).
//
// One CTA owns a TW x TH tile of elements, NG1 = p + 2 (p = 1: 2) threads per element.
//   load    the tile's nodal state (TMA, or plain coalesced loads) and the face-node strips of the
//           neighbours on its four edges -> shared memory
//   volume  thread (element, column gx): contracts its column in x, forms the point fluxes of its
//           NG1 points and lifts them in y: the column sums Ax, Ay (x / y fluxes) and As (the alpha
//           source) of every y-node, kept in registers, then in shared memory
//   faces   one thread per face of the tile: both traces, the Riemann fluxes of its p + 1 points
//           and their lift along the face, once per face
//   update  thread (element, field, y-node): lifts the column sums in x, adds the four faces'
//           shares and applies the stage update to its p + 1 nodes (coalesced)
// The inverse mass matrix M^-1 = (1/J) M1^-1 (x) M1^-1, the quadrature weights and the metric are
// folded into the lift tables (ColTab), so no pass over the nodes is spent on them.
// Tiles at the right and top edges of grids whose extents are not tile multiples are cut: their
// last column / row is where the right / top neighbours' strips and boundary rules apply.
// Equivalent to DG_SOLVER::dg_solver (code/src/dg/dg_solver.h:292-364) + Lsolver + the RK register
// update, up to FP64 rounding.
#pragma once
#include "common.cuh"
#include "physics.cuh"
#include "tma.cuh"

namespace dgb {

// Tables of one problem (1D factors; rows padded to the largest order), passed by value: they are
// read as constant-bank operands.
struct ColTab {
  double B1[MAXG][MAXN];            // l_i(x_g)
  double Dx[MAXG][MAXN], Dy[MAXG][MAXN];  // 2/hx l'_i(x_g), 2/hy l'_i(x_g)  (gradient of alpha)
  double LB[MAXG][MAXN], LD[MAXG][MAXN];  // w_g (M1^-1 l)(x_g), w_g (M1^-1 l')(x_g)  (lift in y)
  double XD[MAXG][MAXN], XB[MAXG][MAXN], XS[MAXG][MAXN];  // lift in x of Ax, Ay, As, metric included
  double BF[MAXN][MAXN];            // l_j on the face's Gauss points
  double LF[MAXN][MAXN];            // 1/2 wf_g (M1^-1 l)(xf_g): face lift (the fluxes come doubled)
  double EX[2][MAXN], EY[2][MAXN];  // M1^-1 column of the first / last node, face metric and sign
};

// One stage of one problem
struct ColArgs {
  const double* __restrict__ U;     // stage input
  const double* base;               // out = k0 base + k1 U + k2 du   (base not read when k0 == 0;
  double* out;                      //   it may be `out` itself)
  const double* base2;              // out2 = base2 + c2 du           (out2 null: not formed)
  double* out2;
  const int* __restrict__ nbr;
  const DevScalars* __restrict__ scal;
  unsigned int* errflag;            // receives FLAG_TIMEOUT when a bounded wait runs out
  long long polls;                  // budget of the first wait on each tile copy (then drained)
  double k0, k1, k2, c2;
  double dt;                        // du = dt M^-1 (...); 0: the step in scal
  double sx, sy;                    // SCALED: 2/hx, 2/hy (the tables are those of hx = hy = 2)
  int nx, ny, ld, tma;
};

// Shapes.  The kernel is bound by instruction issue and latency, not by bandwidth: of some 7,300
// instructions per p = 2 element 3,200 are FP64 (20 us of a full FP64 pipe per 512 x 256 launch).  With
// one thread per element the 45 nodal accumulators and the column sums do not fit 255 registers, 8 warps
// per SM are resident and they spill: 84 us.  Split over the quadrature columns a thread needs 128
// registers, 16 warps are resident, and what the columns exchange is the y-lifted sums (27 per column
// at p = 2), not the nodes.  Measured per launch (Rusanov, the launch of one thread per element first):
//   p = 1, 1000 x 500   126 us; tiles 16 x 8: 89, 16 x 4: 84, 32 x 4: 87, 16 x 2: 93, 8 x 4: 99
//   p = 2, 512 x 256     84 us; 16 x 4: 54, 16 x 2: 52, 32 x 2: 55, 8 x 4: 56, 8 x 8: 59
//   p = 3, 1024 x 512   888 us; 16 x 2: 450, 8 x 4: 437, 16 x 4: 479, 32 x 2: 493, 8 x 8: 491   (Roe)
// Small tiles pay more faces per element (16 x 4: 2.31, 16 x 2: 2.56) but put more CTAs on an SM, whose
// loads, barriers and compute phases then overlap.  With the step's status read beside the tile's copy instead of
// before it, the stage base prefetched into L2 and 32-bit offsets: 50 us (p = 2), 421 us (p = 3).  There it
// spends 10 us on the volume terms, 10 on the faces, 13 on the update and 20 on loads, in p = 2's 50 (the
// copy rate would take 22 for stages 2 and 3); starting the CTAs of an SM staggered changes nothing.
template <int P>
constexpr int col_tw() { return P == 3 ? 8 : 16; }
template <int P>
constexpr int col_th() { return P == 2 ? 2 : 4; }
template <int P, int NY, bool GC, int TW_ = col_tw<P>(), int TH_ = col_th<P>()>
struct ColDims {
  static constexpr int N1 = P + 1, NS = N1 * N1, NF = 5 + NY, NG1 = P == 1 ? 2 : P + 2;
  static constexpr int NFL = 4 + NY + (GC ? 1 : 0);       // fields with a conservative volume flux
  static constexpr int NA = (2 * NFL + (GC ? 0 : 1)) * N1;  // column sums per thread
  static constexpr int TW = TW_, TH = TH_;
  static constexpr int NE = TW * TH, NT = NE * NG1;
  static constexpr int NXF = (TW + 1) * TH, NYF = TW * (TH + 1), NFACE = NXF + NYF;
  static constexpr int NEDGE = 2 * TH + 2 * TW;           // edge slots: left, right, bottom, top
  static constexpr size_t off_code = 128;
  static constexpr size_t off_tile = off_code + (NEDGE * 4 + 127) / 128 * 128;
  static constexpr size_t tile_bytes = sizeof(double) * NF * NS * NE;
  static constexpr size_t off_halo = off_tile + tile_bytes;
  static constexpr size_t off_face = off_halo + sizeof(double) * NF * N1 * NEDGE;
  static constexpr size_t off_sums = off_face + sizeof(double) * (NF + 1) * N1 * NFACE;
  static constexpr size_t smem_bytes = off_sums + sizeof(double) * NA * NT;
  // CTAs per SM: what the shared memory (227 KB, 1 KB of it reserved per CTA) and 64 K registers hold
  static constexpr int by_smem = (int)(227 * 1024 / (smem_bytes + 1024));
  static constexpr int want_regs = P == 1 ? 96 : P == 2 ? 128 + 24 * (NY + (GC ? 1 : 0)) : 168 + 24 * NY;
  static constexpr int by_regs = 65536 / (NT * (want_regs > 255 ? 255 : want_regs));
  static constexpr int ctas = by_smem < 1 || by_regs < 1 ? 1 : (by_smem < by_regs ? by_smem : by_regs);
  static_assert(NE % 32 == 0, "a warp shares its quadrature column and field");
};

// Doubled Riemann flux in the face's frame: states (rho, m_n, m_t, E, alpha | rho Y), normal +1.
// F2 = 2 F, nc2 = 2 ncterm of phys::riemann2d_rcp.
template <int FLUX, int NY, bool GC>
__device__ __forceinline__ void riemann_n2(const double* L, const double* R, double* F2, double& nc2) {
  const double rL = L[0], rR = R[0];
  const double irL = phys::rcp(rL), irR = phys::rcp(rR);
  const double nL = L[1] * irL, tL = L[2] * irL, nR = R[1] * irR, tR = R[2] * irR;
  // GAMCONS: alpha = field / rho; the reference's Rusanov solver takes its right alpha from the left
  // state, divided twice (twod_multifluid_fluxes.h:50-53)
  const double aL = GC ? L[4] * irL : L[4];
  const double aR = GC ? (FLUX == phys::FLUX_ROE ? R[4] * irR : aL * irL) : R[4];
  const double gL = phys::rcp(aL), gR = phys::rcp(aR);  // gamma - 1
  const double EL = L[3], ER = R[3];
  const double pL = gL * (EL - 0.5 * (L[1] * nL + L[2] * tL));
  const double pR = gR * (ER - 0.5 * (R[1] * nR + R[2] * tR));
  if constexpr (FLUX == phys::FLUX_ROE) {
    const double HL = (EL + pL) * irL, HR = (ER + pR) * irR;
    const double iL = pL * aL, iR = pR * aR;
    const double RT = phys::root(rR * irL), i1 = phys::rcp(1 + RT), rho = RT * rL;
    const double vn = (nL + RT * nR) * i1, vt = (tL + RT * tR) * i1, H = (HL + RT * HR) * i1;
    const double alpha = (aL + RT * aR) * i1, gm1 = phys::rcp(alpha);
    const double ke = 0.5 * (vn * vn + vt * vt);
    const double a = phys::root(gm1 * (H - ke)), ia = phys::rcp(a);
    const double i = (iL + RT * iR) * i1, p = gm1 * i;
    const double dal = aR - aL;
    const double dp = gm1 * gm1 * (alpha * (iR - iL) - i * dal);
    const double ia2 = ia * ia, h2a = 0.5 * ia2, rad = rho * a * (nR - nL);
    const double dV0 = (dp - rad) * h2a, dV1 = rho * (tR - tL) * ia, dV2 = (rR - rL) - dp * ia2, dV3 = (dp + rad) * h2a;
    const double ws1 = fabs(vn);
    const double w0 = fabs(vn - a) * dV0, w1 = ws1 * dV1, w2 = ws1 * dV2, w3 = fabs(vn + a) * dV3, w4 = ws1 * dal;
    const double wa = w1 * a, ws = w0 + w2 + w3, wd = (w3 - w0) * a;
    F2[0] = (L[1] + R[1]) - ws;
    F2[1] = ((L[1] * nL + pL) + (R[1] * nR + pR)) - (ws * vn + wd);
    F2[2] = (L[1] * tL + R[1] * tR) - (ws * vt + wa);
    F2[3] = (L[1] * HL + R[1] * HR) - ((w0 + w3) * H + wd * vn + wa * vt + w2 * ke + w4 * p);
    F2[4] = GC ? (rL * nL * aL + rR * nR * aR) - w4 : -w4;
    nc2 = GC ? 0.0 : -vn * dal;
#pragma unroll
    for (int k = 0; k < NY; ++k) {
      const double Y = (L[5 + k] * irL + RT * R[5 + k] * irR) * i1;
      const double dVY = R[5 + k] - L[5 + k] - (dV0 + dV2 + dV3) * Y;
      F2[5 + k] = (L[5 + k] * nL + R[5 + k] * nR) - (ws * Y + ws1 * dVY);
    }
  } else {
    const double cL = phys::root((1.0 + gL) * pL * irL), cR = phys::root((1.0 + gR) * pR * irR);
    const double s = fmax(fabs(nL) + cL, fabs(nR) + cR);
    F2[0] = (L[1] + R[1]) - s * (rR - rL);
    F2[1] = ((L[1] * nL + pL) + (R[1] * nR + pR)) - s * (R[1] - L[1]);
    F2[2] = (L[1] * tL + R[1] * tR) - s * (R[2] - L[2]);
    F2[3] = ((EL + pL) * nL + (ER + pR) * nR) - s * (ER - EL);
    if (GC) {
      F2[4] = (rL * nL * aL + rR * nR * aR) - s * (rR * aR - rL * aL);
      nc2 = 0.0;
    } else {
      const double dal = aR - aL;
      F2[4] = -s * dal;
      nc2 = -0.5 * (nL + nR) * dal;
    }
    // the reference's mass-fraction line has its dissipation outside the 1/2 (fluxes.h:91-94)
#pragma unroll
    for (int k = 0; k < NY; ++k) F2[5 + k] = (L[5 + k] * nL + R[5 + k] * nR) - 2.0 * (s * (R[5 + k] - L[5 + k]));
  }
}

// The tile (origin tx0, ty0; tw x th elements of it) and the neighbours' face nodes into shared memory.  The caller
// has initialised the mbarrier at its start; `phase` counts its completed phases (a persistent caller
// runs many tiles on one barrier).  Returns whether there is work, for the whole CTA, after its last barrier.
template <class Dm, int P>
__device__ __forceinline__ bool cols_load(const ColArgs& a, const CUtensorMap* mapU, const CUtensorMap* mapBase, int tx0,
                                          int ty0, int tw, int th, unsigned char* smraw, uint32_t& phase) {
  constexpr int N1 = Dm::N1, NS = Dm::NS, NF = Dm::NF, NE = Dm::NE, NT = Dm::NT, TW = Dm::TW, TH = Dm::TH;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smraw);
  int* s_ok = reinterpret_cast<int*>(smraw + 8);
  int* codes = reinterpret_cast<int*>(smraw + Dm::off_code);       // [NEDGE] neighbours / boundary codes
  double* Us = reinterpret_cast<double*>(smraw + Dm::off_tile);    // [NF*NS][NE]
  double* HS = reinterpret_cast<double*>(smraw + Dm::off_halo);    // [NF*N1][NEDGE] neighbours' face nodes
  const int tid = threadIdx.x, ld = a.ld, nx = a.nx;
  const double* U = after_wait(a.U);
  // (the step's status is read along with them: its latency before the copy would be every CTA's)
  const unsigned failed = tid == 0 && a.scal ? ld_dep(&a.scal->flags) : 0u;
  // a TMA copy must land on a 128-byte shared boundary and start on a 16-byte global column;
  // otherwise record the fault and skip the copy
  const bool tma_ok = a.tma && (smem_u32(Us) & 127u) == 0 && ((tx0 * 8) & 15) == 0;
  if (tid == 0) {
    if (tma_ok) {
      mbar_arrive_expect_tx(bar, (uint32_t)Dm::tile_bytes);
      tma_load_3d(Us, mapU, tx0, ty0, 0, bar);
      if (a.k0 != 0.0 && mapBase) tma_prefetch_3d(mapBase, tx0, ty0, 0);
    } else if (a.tma) {
      atomicOr(a.errflag, (unsigned)FLAG_TIMEOUT);
    }
  }
  if (!a.tma) {
    for (int k = tid; k < NF * NS * NE; k += NT) {
      const int q = k / NE, el = k % NE, x = el % TW, y = el / TW;
      Us[k] = x < tw && y < th ? ld_after(U + (size_t)q * ld + (size_t)(ty0 + y) * nx + tx0 + x) : 0.0;
    }
  }
  // edge slot s of the tile (left, right, bottom, top): the neighbour across it -- the next element of the row or
  // column, or at the domain's edges what the neighbour table says -- and its face nodes.  A thread takes
  // node j of every field of one slot, all loads in flight.  (Offsets into a state are 32-bit counts of
  // values: dgb_create refuses larger states.)
  const unsigned plane = ld;
  for (int k = tid; k < N1 * Dm::NEDGE; k += NT) {
    const int s = k % Dm::NEDGE, j = k / Dm::NEDGE;
    const bool side = s < 2 * TH;
    const int hi = side ? s / TH : (s - 2 * TH) / TW, q = side ? s % TH : (s - 2 * TH) % TW;
    if (q < (side ? th : tw)) {
      const int x = side ? tx0 + (hi ? tw - 1 : 0) : tx0 + q, y = side ? ty0 + q : ty0 + (hi ? th - 1 : 0);
      const int eo = y * nx + x;
      const bool border = side ? (hi ? x == nx - 1 : x == 0) : (hi ? y == a.ny - 1 : y == 0);
      const int step = side ? 1 : nx;
      const int nb = border ? __ldg(a.nbr + (size_t)(side ? hi : 2 + hi) * ld + eo) : (hi ? eo + step : eo - step);
      const unsigned o = ((side ? (hi ? 0 : P) : (hi ? 0 : N1 * P)) + (side ? N1 : 1) * j) * plane + (unsigned)nb;
      double v[NF];
#pragma unroll
      for (int f = 0; f < NF; ++f) v[f] = nb >= 0 ? ld_after(U + (o + f * NS * plane)) : 0.0;
      if (j == 0) codes[s] = nb;
#pragma unroll
      for (int f = 0; f < NF; ++f) HS[(f * N1 + j) * Dm::NEDGE + s] = v[f];
    }
  }
  if (tid == 0) {
    bool ok = !a.tma || (tma_ok && mbar_wait(bar, phase & 1, a.polls));
    if (tma_ok && !ok) {
      atomicOr(a.errflag, (unsigned)FLAG_TIMEOUT);
      mbar_wait(bar, phase & 1);
    }
    *s_ok = ok && !failed ? 1 : 0;
  }
  if (tma_ok) ++phase;
  __syncthreads();
  return *s_ok != 0;
}

// The work of one tile (origin tx0, ty0).
// SCALED: the tables carry no metric, a.sx and a.sy do (tiles of problems of many mesh widths).
template <int P, int FLUX, int NY, bool GC, int TW, int TH, bool SCALED>
__device__ __forceinline__ void cols_body(const ColArgs& a, const ColTab& tab, const CUtensorMap* mapU,
                                          const CUtensorMap* mapBase, int tx0, int ty0, unsigned char* smraw,
                                          uint32_t& phase) {
  static_assert(!(GC && NY > 0), "GAMCONS with mass fractions is not built");
  using Dm = ColDims<P, NY, GC, TW, TH>;
  constexpr int N1 = Dm::N1, NS = Dm::NS, NF = Dm::NF, NFL = Dm::NFL, NG1 = Dm::NG1;
  constexpr int NE = Dm::NE, NT = Dm::NT, NXF = Dm::NXF, NFACE = Dm::NFACE;
  int* codes = reinterpret_cast<int*>(smraw + Dm::off_code);       // [NEDGE] neighbours / boundary codes
  double* Us = reinterpret_cast<double*>(smraw + Dm::off_tile);    // [NF*NS][NE]
  double* HS = reinterpret_cast<double*>(smraw + Dm::off_halo);    // [NF*N1][NEDGE] neighbours' face nodes
  double* FS = reinterpret_cast<double*>(smraw + Dm::off_face);    // [(NF+1)*N1][NFACE] lifted face fluxes
  double* AS = reinterpret_cast<double*>(smraw + Dm::off_sums);    // [NA][NT] column sums
  const int tid = threadIdx.x, ld = a.ld, nx = a.nx;
  const int tw = min(TW, nx - tx0), th = min(TH, a.ny - ty0);

  if (!cols_load<Dm, P>(a, mapU, mapBase, tx0, ty0, tw, th, smraw, phase)) return;
  const unsigned plane = ld;

  // ---------------- volume: one thread per (element, quadrature column) ----------------
  {
    const int el = tid % NE, gx = tid / NE;
    if (el % TW < tw && el / TW < th) {
      double T[NF][N1], dT[N1];  // column values: sum_ix l_ix(x_gx) u(ix, iy), and of 2/hx l' for alpha
      {
        double b[N1], d[N1];
#pragma unroll
        for (int ix = 0; ix < N1; ++ix) { b[ix] = tab.B1[gx][ix]; d[ix] = SCALED ? a.sx * tab.Dx[gx][ix] : tab.Dx[gx][ix]; }
#pragma unroll
        for (int iy = 0; iy < N1; ++iy) {
#pragma unroll
          for (int f = 0; f < NF; ++f) {
            double u = Us[(f * NS + N1 * iy) * NE + el];
            T[f][iy] = b[0] * u;
            if (!GC && f == 4) dT[iy] = d[0] * u;
#pragma unroll
            for (int ix = 1; ix < N1; ++ix) {
              u = Us[(f * NS + ix + N1 * iy) * NE + el];
              T[f][iy] += b[ix] * u;
              if (!GC && f == 4) dT[iy] += d[ix] * u;
            }
          }
        }
      }
      double Ax[NFL][N1], Ay[NFL][N1], As[N1];
#pragma unroll
      for (int gy = 0; gy < NG1; ++gy) {
        double ug[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
          ug[f] = tab.B1[gy][0] * T[f][0];
#pragma unroll
          for (int iy = 1; iy < N1; ++iy) ug[f] += tab.B1[gy][iy] * T[f][iy];
        }
        // volume flux and alpha source (evaluate_sf, code/src/physics/physics.cu:248-301)
        const double rho = ug[0], ir = phys::rcp(rho), ia = phys::rcp(ug[4]);
        const double gm1 = GC ? rho * ia : ia;
        const double u = ug[1] * ir, v = ug[2] * ir;
        const double p = gm1 * (ug[3] - 0.5 * (ug[1] * u + ug[2] * v));
        const double H = ug[3] + p;
        double fx[NFL], fy[NFL];
        fx[0] = ug[1]; fx[1] = ug[1] * u + p; fx[2] = ug[2] * u; fx[3] = H * u;
        fy[0] = ug[2]; fy[1] = fx[2]; fy[2] = ug[2] * v + p; fy[3] = H * v;
#pragma unroll
        for (int k = 4; k < NFL; ++k) { fx[k] = ug[GC ? k : k + 1] * u; fy[k] = ug[GC ? k : k + 1] * v; }
#pragma unroll
        for (int iy = 0; iy < N1; ++iy) {
#pragma unroll
          for (int f = 0; f < NFL; ++f) {
            if (gy == 0) {
              Ax[f][iy] = tab.LB[0][iy] * fx[f];
              Ay[f][iy] = tab.LD[0][iy] * fy[f];
            } else {
              Ax[f][iy] += tab.LB[gy][iy] * fx[f];
              Ay[f][iy] += tab.LD[gy][iy] * fy[f];
            }
          }
        }
        if constexpr (!GC) {
          double dax = tab.B1[gy][0] * dT[0], day = tab.Dy[gy][0] * T[4][0];
#pragma unroll
          for (int iy = 1; iy < N1; ++iy) { dax += tab.B1[gy][iy] * dT[iy]; day += tab.Dy[gy][iy] * T[4][iy]; }
          if (SCALED) day *= a.sy;
          const double src = -(u * dax + v * day);
#pragma unroll
          for (int iy = 0; iy < N1; ++iy) As[iy] = gy == 0 ? tab.LB[0][iy] * src : As[iy] + tab.LB[gy][iy] * src;
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

  // ---------------- faces: one thread per face of the tile ----------------
  // x-faces (row, column 0..TW) then y-faces (row 0..TH, column); the left / bottom element is L.  At a
  // domain boundary the inside element is L with its outward normal and its mirror image R
  // (reflective walls mirror the wall-normal momentum, code/src/bc/boundaries.cu:20-67); on the left
  // and bottom sides that is computed in the reversed frame and stored with the sign of +x / +y.
  for (int fc = tid; fc < NFACE; fc += NT) {
    const bool xf = fc < NXF;
    const int k = xf ? fc : fc - NXF;
    const int fx = xf ? k % (TW + 1) : k % TW, fy = xf ? k / (TW + 1) : k / TW;
    if (xf ? (fx > tw || fy >= th) : (fx >= tw || fy > th)) continue;
    const int pos = xf ? fx : fy, last = xf ? tw : th;
    // offsets of node j of field f: o + f * sf + j * sj (in Us, or in HS for an edge slot)
    const int sj = xf ? N1 * NE : NE;
    const int slot = xf ? (pos == 0 ? fy : TH + fy) : 2 * TH + (pos == 0 ? 0 : TW) + fx;
    const bool edge = pos == 0 || pos == last;
    const int code = edge ? codes[slot] : 0;
    const int elR = fy * TW + fx, elL = xf ? elR - 1 : elR - TW;
    const double* pL = Us + (xf ? P : N1 * P) * NE + elL;
    const double* pR = Us + elR;
    int sfL = NS * NE, sjL = sj, sfR = NS * NE, sjR = sj;
    if (pos == 0) { pL = HS + slot; sfL = N1 * Dm::NEDGE; sjL = Dm::NEDGE; }
    else if (pos == last) { pR = HS + slot; sfR = N1 * Dm::NEDGE; sjR = Dm::NEDGE; }
    const bool flip = code < 0 && pos == 0;
    if (code < 0) {  // both sides read the inside element
      if (pos == 0) { pL = pR; sfL = sfR; sjL = sjR; }
      else { pR = pL; sfR = sfL; sjR = sjL; }
    }
    const int fn = xf ? 1 : 2, ft = xf ? 2 : 1;  // normal and tangential momentum
    double tl[NF][N1], tr[NF][N1];
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const int ff = f == 1 ? fn : f == 2 ? ft : f;
      double vl[N1], vr[N1];
#pragma unroll
      for (int j = 0; j < N1; ++j) { vl[j] = pL[ff * sfL + j * sjL]; vr[j] = pR[ff * sfR + j * sjR]; }
#pragma unroll
      for (int g = 0; g < N1; ++g) {
        tl[f][g] = tab.BF[g][0] * vl[0];
        tr[f][g] = tab.BF[g][0] * vr[0];
#pragma unroll
        for (int j = 1; j < N1; ++j) { tl[f][g] += tab.BF[g][j] * vl[j]; tr[f][g] += tab.BF[g][j] * vr[j]; }
      }
    }
    if (code < 0) {
#pragma unroll
      for (int g = 0; g < N1; ++g) {
        if (flip) { tl[1][g] = -tl[1][g]; tr[1][g] = -tr[1][g]; }
        if (code == -3) tr[1][g] = -tr[1][g];
      }
    }
    double Ff[NF + 1][N1];  // lifted along the face; fields, then alpha as its left-hand element sees it
#pragma unroll
    for (int g = 0; g < N1; ++g) {
      double L[NF], R[NF], F2[NF], nc2;
#pragma unroll
      for (int f = 0; f < NF; ++f) { L[f] = tl[f][g]; R[f] = tr[f][g]; }
      riemann_n2<FLUX, NY, GC>(L, R, F2, nc2);
      const double am = F2[4] - nc2;
      F2[4] += nc2;
#pragma unroll
      for (int f = 0; f <= NF; ++f)
#pragma unroll
        for (int j = 0; j < N1; ++j) {
          const double v = f < NF ? F2[f < NF ? f : 0] : am;
          Ff[f][j] = g == 0 ? tab.LF[0][j] * v : Ff[f][j] + tab.LF[g][j] * v;
        }
    }
    if (flip) {  // -F with the same nc: the two alpha records trade places
#pragma unroll
      for (int j = 0; j < N1; ++j) {
#pragma unroll
        for (int f = 0; f < NF; ++f)
          if (f != 1 && f != 4) Ff[f][j] = -Ff[f][j];
        const double ap = Ff[4][j];
        Ff[4][j] = -Ff[NF][j];
        Ff[NF][j] = -ap;
      }
    }
#pragma unroll
    for (int f = 0; f <= NF; ++f) {
      const int ff = f == 1 ? fn : f == 2 ? ft : f;
#pragma unroll
      for (int j = 0; j < N1; ++j) FS[(ff * N1 + j) * NFACE + fc] = Ff[f][j];
    }
  }
  // ---------------- update: one thread per (element, field, y-node) ----------------
  // (the stage base and the accumulator are read before the barrier: their latency passes while the
  // other warps finish)
  // Item r = field * N1 + y-node: column sums at slots r (x) and NFL * N1 + r (y) of AS -- past alpha,
  // which has none under GAMNCON, N1 less --, face records at r, nodes from plane N1 * r.
  constexpr int NIT = (NF * N1 + NG1 - 1) / NG1;
  const int el = tid % NE, tx = el % TW, ty = el / TW, r0 = tid / NE;
  const bool own = tx < tw && ty < th;
  const unsigned g0 = N1 * r0 * plane + (unsigned)((ty0 + ty) * nx + tx0 + tx);
  const double *base = after_wait(a.base), *base2 = after_wait(a.base2);
  double v0[NIT][N1], v2[NIT][N1];
#pragma unroll
  for (int q = 0; q < NIT; ++q) {
    const bool on = own && r0 + q * NG1 < NF * N1;
#pragma unroll
    for (int ix = 0; ix < N1; ++ix) {
      const unsigned gi = g0 + (q * NG1 * N1 + ix) * plane;
      v0[q][ix] = on && a.k0 != 0.0 ? ld_after(base + gi) : 0.0;
      v2[q][ix] = on && a.out2 ? ld_after(base2 + gi) : 0.0;
    }
  }
  const double dt = a.dt > 0 ? a.dt : ld_dep(&a.scal->dt);
  __syncthreads();
  if (own) {
    const double* fx = FS + r0 * NFACE + ty * (TW + 1) + tx;
#pragma unroll
    for (int q = 0; q < NIT; ++q) {
      const int r = r0 + q * NG1;
      if ((q + 1) * NG1 > NF * N1 && r >= NF * N1) break;
      const bool alpha = q * NG1 + NG1 > 4 * N1 && q * NG1 < 5 * N1 && r >= 4 * N1 && r < 5 * N1;
      const int iy = r % N1;
      double s[N1];
      if (!GC && alpha) {
        const double* as = AS + (2 * NFL * N1 - 4 * N1 + r) * NT + el;
#pragma unroll
        for (int gx = 0; gx < NG1; ++gx) {
          const double v = as[gx * NE];
#pragma unroll
          for (int ix = 0; ix < N1; ++ix) s[ix] = gx == 0 ? tab.XS[0][ix] * v : s[ix] + tab.XS[gx][ix] * v;
        }
      } else {
        const double* as = AS + (GC || NY == 0 || r < 4 * N1 ? r : r - N1) * NT + el;
#pragma unroll
        for (int gx = 0; gx < NG1; ++gx) {
          double vx = as[gx * NE], vy = as[NFL * N1 * NT + gx * NE];
          if (SCALED) { vx *= a.sx; vy *= a.sy; }
#pragma unroll
          for (int ix = 0; ix < N1; ++ix) {
            s[ix] = gx == 0 ? tab.XD[0][ix] * vx : s[ix] + tab.XD[gx][ix] * vx;
            s[ix] += tab.XB[gx][ix] * vy;
          }
        }
      }
      {
        const int far = alpha ? (NF - 4) * N1 * NFACE : 0;  // the record the element left of / below a face reads
        double l = fx[q * NG1 * NFACE], rr = fx[q * NG1 * NFACE + 1 + far];
        const double* fy = FS + (r - iy) * NFACE + NXF + el;
        double eb = tab.EY[0][iy], et = tab.EY[1][iy];
        if (SCALED) { l *= a.sx; rr *= a.sx; eb *= a.sy; et *= a.sy; }
#pragma unroll
        for (int ix = 0; ix < N1; ++ix)
          s[ix] += tab.EX[0][ix] * l + tab.EX[1][ix] * rr + eb * fy[ix * NFACE] + et * fy[ix * NFACE + TW + far];
      }
      const double* us = Us + N1 * r * NE + el;
#pragma unroll
      for (int ix = 0; ix < N1; ++ix) {
        const unsigned gi = g0 + (q * NG1 * N1 + ix) * plane;
        const double du = dt * s[ix];
        double o = a.k2 * du;
        if (a.k1 != 0.0) o = a.k1 * us[ix * NE] + o;
        if (a.k0 != 0.0) o = a.k0 * v0[q][ix] + o;
        a.out[gi] = o;
        if (a.out2) a.out2[gi] = v2[q][ix] + a.c2 * du;
      }
    }
  }
}

template <int P, int FLUX, int NY, bool GC>
__global__ void __launch_bounds__(ColDims<P, NY, GC>::NT, ColDims<P, NY, GC>::ctas)
    residual2d_cols_kernel(const __grid_constant__ ColArgs a, const __grid_constant__ ColTab tab,
                           const __grid_constant__ CUtensorMap mapU, const __grid_constant__ CUtensorMap mapBase) {
  constexpr int TW = col_tw<P>(), TH = col_th<P>();
  extern __shared__ __align__(128) unsigned char smraw[];
  if (threadIdx.x == 0) {
    mbar_init(reinterpret_cast<uint64_t*>(smraw), 1);
    fence_mbar_init();
  }
  pdl_wait();
  const int ty0 = tile_row() * TH;
  if (ty0 >= a.ny) return;
  uint32_t phase = 0;
  cols_body<P, FLUX, NY, GC, TW, TH, false>(a, tab, &mapU, &mapBase, blockIdx.x * TW, ty0, smraw, phase);
  // (at the end: with the trigger at the start the next launch's CTAs, waiting, hold the shared memory that this
  // one's last wave could use: 240 -> 256 us per 512 x 256 step)
  pdl_trigger();
}

}  // namespace dgb
