// 2D limiters of structured row-major grids (HR and m2 methods).
//
//   lim2d_kernel       both passes in one launch, out of place: one thread per element and slice (its body also
//                      limits the batched ensemble)
//   lim2d_*pass_*      x pass, then y pass through a global scratch: the allocation-free limiter, primitive
//                      variables, more than three mass fractions
//
// Either way every element's moments (hr_moments) are computed once per slice and shared with the
// neighbours that need them.
//   x pass: CTA = 30 consecutive elements of one element row (+ left/right neighbour slots),
//           threads (element slot, y-slice)
//   y pass: CTA = 32 x 4 elements (+ bottom/top neighbour rows), threads (x slot, row slot),
//           one x-column of nodes per CTA (grid z)
// Output of the x pass (global scratch X): m2 -> [rho, rhou, rhov, alpha, p, E],
// HR -> the five conserved fields, all x-limited and in Lagrange form (limiting.cc:271-409).
#pragma once
#include "kernels.cuh"

namespace dgb {

// Dynamic shared memory of the tiled limiter passes: 0 while their per-quantity arrays fit the
// static limit (up to three mass fractions), else the arrays' size
template <int P, int NY>
constexpr size_t lim2d_xpass_smem_bytes() {
  const size_t b = sizeof(double) * (5 + NY) * (P + 1) * Hr2<P>::NM * 32;
  return b <= 48 * 1024 ? 0 : b;
}
template <int P, int NY>
constexpr size_t lim2d_ypass_smem_bytes() {
  const size_t b = sizeof(double) * (5 + NY) * Hr2<P>::NM * 6 * 32;
  return b <= 48 * 1024 ? 0 : b;
}

// x pass over one block of the row ey starting at element column x0 (a multiple of 30); the CTA
// returns from here together, after its last barrier
// NY mass fractions: limited like the density (m2: the MACRO blocks of M2limiting,
// limiting.cc:327-331 and 398-404; HR: every field); in X after E (m2) or as fields (HR).
template <int P, int METHOD, int NY = 0>
__device__ __forceinline__ void lim2d_xpass_body(const LimArgs la, int nx, const double* __restrict__ U,
                                                 const int* __restrict__ nbr, double* __restrict__ X, int x0,
                                                 int ey) {
  constexpr int N1 = P + 1, NS = N1 * N1, NQ = 5 + NY, NF = 5 + NY, TWI = 30;
  using HR = Hr2<P>;
  constexpr int NM = HR::NM;
  // [quantity][slice][moment][slot]: static shared memory, or dynamic (lim2d_xpass_smem_bytes)
  // when the quantities would not fit the static limit (many mass fractions)
  double(*A)[N1][NM][32];
  if constexpr (lim2d_xpass_smem_bytes<P, NY>() == 0) {
    __shared__ double As[NQ][N1][NM][32];
    A = As;
  } else {
    extern __shared__ __align__(16) double lsm[];
    A = reinterpret_cast<double(*)[N1][NM][32]>(lsm);
  }
  const int ld = la.ld;
  const int tx = threadIdx.x, sl = threadIdx.y;
  const int ex = x0 - 1 + tx;
  // element held by this slot: interior element, or the neighbour of the adjacent interior one
  const bool interior = tx >= 1 && tx <= TWI && ex < nx;
  int e = -1;
  if (interior) e = ey * nx + ex;
  else if (tx == 0) e = __ldg(nbr + (size_t)0 * ld + ey * nx + x0);
  else if (ex - 1 < nx && ex - 1 >= 0) e = __ldg(nbr + (size_t)1 * ld + ey * nx + ex - 1);
  double v[NF][N1], q[NQ][N1];
  if (e >= 0) {
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
      for (int ix = 0; ix < N1; ++ix) v[f][ix] = ld_after(U + (size_t)(f * NS + ix + N1 * sl) * ld + e);
#pragma unroll
    for (int ix = 0; ix < N1; ++ix) {
#pragma unroll
      for (int k = 5; k < NQ; ++k) q[k][ix] = v[k][ix];
      if constexpr (METHOD == 1) {
#pragma unroll
        for (int f = 0; f < 5; ++f) q[f][ix] = v[f][ix];
      } else {
        q[0][ix] = v[0][ix];
        q[1][ix] = v[1][ix];
        q[2][ix] = v[2][ix];
        q[3][ix] = v[4][ix];
        // pressure from the unlimited state (pressure kernel, physics.cu:891-958), with reciprocals in place of
        // its divisions
        const double ru = v[1][ix], rv = v[2][ix];
        q[4][ix] = HR::rcp(v[4][ix]) * (v[3][ix] - 0.5 * (ru * ru + rv * rv) * HR::rcp(v[0][ix]));
      }
    }
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      double D[NM];
      HR::moments(q[k], D);
#pragma unroll
      for (int m = 0; m < NM; ++m) A[k][sl][m][tx] = D[m];
    }
  }
  __syncthreads();
  if (!interior) return;
  const int phys = boundary_code(__ldg(nbr + (size_t)0 * ld + e), __ldg(nbr + (size_t)1 * ld + e));
  double lim[NQ][N1];
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    double DL[NM], DC[NM], DR[NM];
#pragma unroll
    for (int m = 0; m < NM; ++m) DC[m] = A[k][sl][m][tx];
    const int ph = (METHOD == 1 && phys == 3 && k == 1) ? 5 : phys;
    if (ph == 0) {
#pragma unroll
      for (int m = 0; m < NM; ++m) { DL[m] = A[k][sl][m][tx - 1]; DR[m] = A[k][sl][m][tx + 1]; }
      HR::limit(DL, DC, DR, q[k], lim[k]);
    } else if (ph == 2 || ph == 3) {
      HR::flat(DC, q[k], lim[k]);
    } else {
      HR::mono(q[k], lim[k]);
    }
  }
  if constexpr (METHOD == 1) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      double out[N1];
      HR::lag(lim[k], out);
#pragma unroll
      for (int ix = 0; ix < N1; ++ix) X[(size_t)(k * NS + ix + N1 * sl) * ld + e] = out[ix];
    }
  } else {
    double r_[N1], u_[N1], v_[N1], a_[N1], p_[N1], K[N1], E_[N1];
    HR::lag(lim[0], r_);
    HR::lag(lim[1], u_);
    HR::lag(lim[2], v_);
    HR::lag(lim[3], a_);
    HR::lag(lim[4], p_);
#pragma unroll
    for (int ix = 0; ix < N1; ++ix) K[ix] = 0.5 * (u_[ix] * u_[ix] + v_[ix] * v_[ix]) * HR::rcp(r_[ix]);
    HR::energy(lim[4], lim[3], K, v[3], E_);
#pragma unroll
    for (int ix = 0; ix < N1; ++ix) {
      const size_t o = (size_t)(ix + N1 * sl) * ld + e;
      X[o + (size_t)0 * NS * ld] = r_[ix];
      X[o + (size_t)1 * NS * ld] = u_[ix];
      X[o + (size_t)2 * NS * ld] = v_[ix];
      X[o + (size_t)3 * NS * ld] = a_[ix];
      X[o + (size_t)4 * NS * ld] = p_[ix];
      X[o + (size_t)5 * NS * ld] = E_[ix];
    }
#pragma unroll
    for (int k = 5; k < NQ; ++k) {
      double y_[N1];
      HR::lag(lim[k], y_);
#pragma unroll
      for (int ix = 0; ix < N1; ++ix) X[(size_t)((k + 1) * NS + ix + N1 * sl) * ld + e] = y_[ix];
    }
  }
}

template <int P, int METHOD, int NY = 0>
__global__ void __launch_bounds__(32 * (P + 1)) lim2d_xpass_tile_kernel(const LimArgs la, int nx,
                                                                      const double* __restrict__ U,
                                                                      const int* __restrict__ nbr,
                                                                      double* __restrict__ X,
                                                                      const DevScalars* __restrict__ scal) {
  pdl_wait();
  if (scal && ld_dep(&scal->flags)) return;
  lim2d_xpass_body<P, METHOD, NY>(la, nx, after_wait(U), nbr, X, blockIdx.x * 30, blockIdx.y);
  pdl_trigger();
}

// y pass over the 32 x 4 element block at (x0, y0) for the node column ix; the CTA returns from
// here together, after its last barrier
template <int P, int METHOD, int NY = 0>
__device__ __forceinline__ void lim2d_ypass_body(const LimArgs la, int nx, int ny, const double* __restrict__ X,
                                                 const int* __restrict__ nbr, double* __restrict__ Uout, int x0,
                                                 int y0, int ix) {
  constexpr int N1 = P + 1, NS = N1 * N1, NQ = 5 + NY, THI = 4;
  using HR = Hr2<P>;
  constexpr int NM = HR::NM;
  // row of quantity k in X: HR -> field k; m2 -> [rho, rhou, rhov, alpha, p, E, rho Y_k]
  auto xrow = [](int k) { return (METHOD == 2 && k >= 5) ? k + 1 : k; };
  // [quantity][moment][row slot][x slot]: static or (many mass fractions) dynamic
  double(*B)[NM][THI + 2][32];
  if constexpr (lim2d_ypass_smem_bytes<P, NY>() == 0) {
    __shared__ double Bs[NQ][NM][THI + 2][32];
    B = Bs;
  } else {
    extern __shared__ __align__(16) double lsm[];
    B = reinterpret_cast<double(*)[NM][THI + 2][32]>(lsm);
  }
  const int ld = la.ld;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int x = x0 + tx;
  const int yy = y0 - 1 + ty;
  const bool interior = ty >= 1 && ty <= THI && yy < ny && x < nx;
  int e = -1;
  if (x < nx) {
    if (interior) e = yy * nx + x;
    else if (ty == 0) e = __ldg(nbr + (size_t)2 * ld + y0 * nx + x);
    else if (yy - 1 < ny && yy - 1 >= 0) e = __ldg(nbr + (size_t)3 * ld + (yy - 1) * nx + x);
  }
  double vE[N1], col[NQ][N1];
  if (e >= 0) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      double D[NM];
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) col[k][iy] = ld_after(X + (size_t)(xrow(k) * NS + ix + N1 * iy) * ld + e);
      HR::moments(col[k], D);
#pragma unroll
      for (int m = 0; m < NM; ++m) B[k][m][ty][tx] = D[m];
    }
    if constexpr (METHOD == 2) {
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) vE[iy] = ld_after(X + (size_t)(5 * NS + ix + N1 * iy) * ld + e);
    }
  }
  __syncthreads();
  if (!interior) return;
  const int phys = boundary_code(__ldg(nbr + (size_t)2 * ld + e), __ldg(nbr + (size_t)3 * ld + e));
  double lim[NQ][N1];
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    double DD[NM], DC[NM], DU[NM];
#pragma unroll
    for (int m = 0; m < NM; ++m) DC[m] = B[k][m][ty][tx];
    const int ph = (METHOD == 1 && phys == 3 && k == 2) ? 5 : phys;
    if (ph == 0) {
#pragma unroll
      for (int m = 0; m < NM; ++m) { DD[m] = B[k][m][ty - 1][tx]; DU[m] = B[k][m][ty + 1][tx]; }
      HR::limit(DD, DC, DU, col[k], lim[k]);
    } else if (ph == 2 || ph == 3) {
      HR::flat(DC, col[k], lim[k]);
    } else {
      HR::mono(col[k], lim[k]);
    }
  }
  if constexpr (METHOD == 1) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      double out[N1];
      HR::lag(lim[k], out);
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) Uout[(size_t)(k * NS + ix + N1 * iy) * ld + e] = out[iy];
    }
  } else {
    double r_[N1], u_[N1], v_[N1], a_[N1], K[N1], E_[N1];
    HR::lag(lim[0], r_);
    HR::lag(lim[1], u_);
    HR::lag(lim[2], v_);
    HR::lag(lim[3], a_);
#pragma unroll
    for (int iy = 0; iy < N1; ++iy) K[iy] = 0.5 * (u_[iy] * u_[iy] + v_[iy] * v_[iy]) * HR::rcp(r_[iy]);
    HR::energy(lim[4], lim[3], K, vE, E_);
#pragma unroll
    for (int iy = 0; iy < N1; ++iy) {
      const size_t o = (size_t)(ix + N1 * iy) * ld + e;
      Uout[o + (size_t)0 * NS * ld] = r_[iy];
      Uout[o + (size_t)1 * NS * ld] = u_[iy];
      Uout[o + (size_t)2 * NS * ld] = v_[iy];
      Uout[o + (size_t)3 * NS * ld] = E_[iy];
      Uout[o + (size_t)4 * NS * ld] = a_[iy];
    }
#pragma unroll
    for (int k = 5; k < NQ; ++k) {
      double y_[N1];
      HR::lag(lim[k], y_);
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) Uout[(size_t)(k * NS + ix + N1 * iy) * ld + e] = y_[iy];
    }
  }
}

template <int P, int METHOD, int NY = 0>
__global__ void __launch_bounds__(32 * 6) lim2d_ypass_tile_kernel(const LimArgs la, int nx, int ny,
                                                                  const double* __restrict__ X,
                                                                  const int* __restrict__ nbr,
                                                                  double* __restrict__ Uout,
                                                                  const DevScalars* __restrict__ scal) {
  pdl_wait();
  if (scal && ld_dep(&scal->flags)) return;
  lim2d_ypass_body<P, METHOD, NY>(la, nx, ny, after_wait(X), nbr, Uout, blockIdx.x * 32, blockIdx.y * 4, blockIdx.z);
  pdl_trigger();
}

}  // namespace dgb

namespace dgb {

// Both limiter passes in one launch, out of place.  A warp is one slice of one element row of the tile,
// a lane one element: 30 elements and the neighbour on either side; ROWS rows and the row below and
// above, P + 1 warps each.  The x pass (warp = y-slice) takes the neighbours' moments by shuffle and leaves
// the x-limited nodes in shared memory; the y pass (warp = x-column) reads its column and those of
// the rows above and below from there, so the x-limited state never goes to memory.  Uout must not alias U.
// Per stage of m2l, against the two passes through a global scratch: p = 2, 512 x 256: 52 -> 33 us; p = 3,
// 1024 x 512: 329 -> 315 (HrTab3's transforms have 16 products, with HrSums it would be 212);
// p = 1, 1024 x 256: 34 -> 23.  The two passes were FP64-bound at half the memory
// rate (2,240 FP64 instructions per p = 2 element, 1,280 now with the halo rows' second x pass) and moved
// 35 B per value; this moves 16 plus halos (15 us at the copy rate) and waits on its loads and its dependent
// operations: 27 warps per SM, issue 55 %, FP64 pipe 34 % (p = 3: 22 warps, 60 %, 54 %).
// Rows per tile: more rows repeat less x work, fewer leave room for a second CTA.  p = 2: 2 rows 41 us,
// 3: 35, 4 (two CTAs): 35, 6: 35, 8: 33; p = 3 (with HrSums): 1: 436, 2: 242, 3: 224, 4: 212; p = 1: 4: 26, 6: 27, 8 (two
// CTAs): 23, 8 (three): 33, 14: 35.  One thread per element with all slices in registers (164
// registers, 12 warps per SM, moments through shared memory) took 39 us at p = 2 and 330 at p = 3.
template <int P, int METHOD, int NY>
struct LimDims {
  static constexpr int NQ = 5 + NY, N1 = P + 1, NX = NQ + (METHOD == 2 ? 1 : 0);  // m2: E after the quantities
  static constexpr int ROWS = P == 3 ? 4 : 8;
  static constexpr int PITCH = 32 * (ROWS + 2), NT = PITCH * N1;
  static constexpr size_t smem_bytes = sizeof(double) * NX * N1 * N1 * PITCH;
  static constexpr int ctas = P == 1 ? 2 : 1;
};

// one tile: element columns from 30 bx, rows from ROWS by
template <int P, int METHOD, int NY>
__device__ __forceinline__ void lim2d_body(const LimArgs la, int nx, int ny, const double* __restrict__ U,
                                           const int* __restrict__ nbr, double* __restrict__ Uout, int bx, int by,
                                           double* lsm) {  // lsm: [quantity, node][row][lane], x-limited nodes
  using Dm = LimDims<P, METHOD, NY>;
  constexpr int N1 = Dm::N1, NS = N1 * N1, NQ = Dm::NQ, NF = 5 + NY, PITCH = Dm::PITCH;
  using HR = Hr2<P>;
  constexpr int NM = HR::NM;
  const int ld = la.ld, tx = threadIdx.x, sl = threadIdx.y, row = threadIdx.z;
  const int ex = bx * 30 - 1 + tx, y = by * Dm::ROWS - 1 + row;
  // the element of column x in this row: beyond the bottom and top sides what the neighbour table says
  auto row_elem = [&](int x) -> int {
    if (y < 0) return __ldg(nbr + (size_t)2 * ld + x);
    if (y == ny) return __ldg(nbr + (size_t)3 * ld + (size_t)(ny - 1) * nx + x);
    return y < ny ? y * nx + x : -1;
  };
  int e = -1;
  if (ex < 0 || ex == nx) {
    const int in = row_elem(ex < 0 ? 0 : nx - 1);
    if (in >= 0) e = __ldg(nbr + (ex < 0 ? 0 : (size_t)ld) + in);
  } else if (ex < nx) {
    e = row_elem(ex);
  }
  const bool icol = tx >= 1 && tx <= 30 && ex < nx;
  double* B = lsm + row * 32 + tx;
  // ---- x pass: the slice iy = sl ----
  {
    double v[NF][N1];
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
      for (int ix = 0; ix < N1; ++ix) v[f][ix] = e >= 0 ? ld_after(U + (size_t)(f * NS + ix + N1 * sl) * ld + e) : 1.0;
    int phx = 0;
    if (e >= 0 && icol && (ex == 0 || ex == nx - 1))
      phx = boundary_code(ex == 0 ? __ldg(nbr + e) : 0, ex == nx - 1 ? __ldg(nbr + (size_t)ld + e) : 0);
    double o[NQ][N1], lp[N1], la_[N1];
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      double q[N1], DC[NM], DL[NM], DR[NM], lim[N1];
#pragma unroll
      for (int ix = 0; ix < N1; ++ix) {
        if (METHOD == 1 || k >= 5) q[ix] = v[k][ix];
        else if (k < 3) q[ix] = v[k][ix];
        else if (k == 3) q[ix] = v[4][ix];
        else  // pressure from the unlimited state (pressure kernel, physics.cu:891-958)
          q[ix] = HR::rcp(v[4][ix]) *
                  (v[3][ix] - 0.5 * (v[1][ix] * v[1][ix] + v[2][ix] * v[2][ix]) * HR::rcp(v[0][ix]));
      }
      HR::moments(q, DC);
#pragma unroll
      for (int m = 0; m < NM; ++m) {
        DL[m] = __shfl_up_sync(0xffffffffu, DC[m], 1);
        DR[m] = __shfl_down_sync(0xffffffffu, DC[m], 1);
      }
      HR::limit(DL, DC, DR, q, lim);
      if (phx != 0) {
        if (phx == 4 || (METHOD == 1 && phx == 3 && k == 1)) HR::mono(q, lim);
        else HR::flat(DC, q, lim);
      }
      HR::lag(lim, o[k]);
#pragma unroll
      for (int ix = 0; ix < N1; ++ix) {
        B[(k * NS + ix + N1 * sl) * PITCH] = o[k][ix];
        if (METHOD == 2 && k == 3) la_[ix] = lim[ix];
        if (METHOD == 2 && k == 4) lp[ix] = lim[ix];
      }
    }
    if constexpr (METHOD == 2) {
      double K[N1], E[N1];
#pragma unroll
      for (int ix = 0; ix < N1; ++ix)
        K[ix] = 0.5 * (o[1][ix] * o[1][ix] + o[2][ix] * o[2][ix]) * HR::rcp(o[0][ix]);
      HR::energy(lp, la_, K, v[3], E);
#pragma unroll
      for (int ix = 0; ix < N1; ++ix) B[(NQ * NS + ix + N1 * sl) * PITCH] = E[ix];
    }
  }
  __syncthreads();
  // ---- y pass: the column ix = sl ----
  if constexpr (P == 3) {  // 16 products per transform: once per column, its Taylor coefficients in place of its nodes
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      double c[N1], A[N1];
      double* b = B + (k * NS + sl) * PITCH;
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) c[iy] = b[N1 * iy * PITCH];
      HR::mono(c, A);
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) b[N1 * iy * PITCH] = A[iy];
    }
    __syncthreads();
  }
  // the moments of what a column of B holds
  auto moments = [](const double* c, double* D) {
    if constexpr (P == 3) HR::means(c, D);
    else HR::moments(c, D);
  };
  if (!icol || row < 1 || row > Dm::ROWS || y >= ny) return;
  int phy = 0;
  if (y == 0 || y == ny - 1)
    phy = boundary_code(y == 0 ? __ldg(nbr + (size_t)2 * ld + e) : 0, y == ny - 1 ? __ldg(nbr + (size_t)3 * ld + e) : 0);
  double* out = Uout + (size_t)sl * ld + e;
  double o[NQ][N1], lp[N1], la_[N1];
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    double c[N1], w[N1], DC[NM], DD[NM], DU[NM], lim[N1];
    const double* b = B + (k * NS + sl) * PITCH;
#pragma unroll
    for (int iy = 0; iy < N1; ++iy) c[iy] = b[N1 * iy * PITCH];
    moments(c, DC);
    if (phy == 0) {
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) w[iy] = b[N1 * iy * PITCH - 32];
      moments(w, DD);
#pragma unroll
      for (int iy = 0; iy < N1; ++iy) w[iy] = b[N1 * iy * PITCH + 32];
      moments(w, DU);
      HR::limit(DD, DC, DU, c, lim);
    } else if (phy == 4 || (METHOD == 1 && phy == 3 && k == 2)) {
      if constexpr (P == 3) {
#pragma unroll
        for (int m = 0; m < N1; ++m) lim[m] = c[m];
      } else {
        HR::mono(c, lim);
      }
    } else {
      HR::flat(DC, c, lim);
    }
    HR::lag(lim, o[k]);
#pragma unroll
    for (int iy = 0; iy < N1; ++iy) {
      const size_t t = (size_t)(N1 * iy) * ld;
      if (METHOD == 1 || k >= 5 || k < 3) out[t + (size_t)k * NS * ld] = o[k][iy];
      else if (k == 3) out[t + (size_t)4 * NS * ld] = o[k][iy];
      if (METHOD == 2 && k == 3) la_[iy] = lim[iy];
      if (METHOD == 2 && k == 4) lp[iy] = lim[iy];
    }
  }
  if constexpr (METHOD == 2) {
    double K[N1], vE[N1], E[N1];
#pragma unroll
    for (int iy = 0; iy < N1; ++iy) {
      vE[iy] = B[(NQ * NS + sl + N1 * iy) * PITCH];
      K[iy] = 0.5 * (o[1][iy] * o[1][iy] + o[2][iy] * o[2][iy]) * HR::rcp(o[0][iy]);
    }
    HR::energy(lp, la_, K, vE, E);
#pragma unroll
    for (int iy = 0; iy < N1; ++iy) out[(size_t)(N1 * iy + 3 * NS) * ld] = E[iy];
  }
}

template <int P, int METHOD, int NY>
__global__ void __launch_bounds__(LimDims<P, METHOD, NY>::NT, LimDims<P, METHOD, NY>::ctas)
    lim2d_kernel(const LimArgs la, int nx, int ny, const double* __restrict__ U, const int* __restrict__ nbr,
                 double* __restrict__ Uout, const DevScalars* __restrict__ scal) {
  extern __shared__ __align__(16) double lsm[];
  pdl_wait();
  if (scal && ld_dep(&scal->flags)) return;
  if (tile_row() * LimDims<P, METHOD, NY>::ROWS >= ny) return;
  lim2d_body<P, METHOD, NY>(la, nx, ny, after_wait(U), nbr, Uout, blockIdx.x, tile_row(), lsm);
  pdl_trigger();
}

}  // namespace dgb
