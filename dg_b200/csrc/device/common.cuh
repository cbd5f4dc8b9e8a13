// Device-side data description shared by all kernels.
//
// Internal state layout ("field-node-major SoA"): U[(f*N_s + t)*ld + e], with
//   f  field, t = ix + (p+1)*iy the tensor-product node index (nodes ascending in x, then y),
//   e  element (mesh order), ld = element count rounded up to a multiple of 64.
// Each (field, node) row is a contiguous run over elements, so a warp touching 32 consecutive
// elements reads 256 contiguous bytes; neighbour traces of a row-major mesh are the same runs
// shifted by +-1 or +-nx.  The reference layout U[(e*N_F+f)*N_s+i] is converted at the API
// boundary only.
#pragma once
#include <cstdint>
#include <type_traits>

namespace dgb {

constexpr int MAXN = 4;    // nodes per direction (p <= 3)
constexpr int MAXG = 5;    // volume quadrature points per direction (p + 2)
constexpr int MAXNS = 16;  // nodes per element

// Small per-problem constants (copied into shared memory by the kernels that index them).
struct Consts {
  int p, n1, ng1, ns, ng, nf, dim;
  int ld, n_elem;
  int pad_;
  // volume quadrature (1D factors): Bq[g][i] = l_i(xq_g), Dq[g][i] = l_i'(xq_g), weights wq
  double Bq[MAXG][MAXN], Dq[MAXG][MAXN], wq[MAXG];
  // face quadrature (p+1 Gauss points): Bf[g][i] = l_i(xf_g), weights wf
  double Bf[MAXN][MAXN], wf[MAXN];
  // element inverse mass matrix in tensor order (Minv[t][t'])
  double Minv[MAXNS][MAXNS];
  // metric of the uniform Cartesian element: J = hx*hy/4 (1D: hx/2), invJac = diag(2/hx, 2/hy)
  double J, ixx, iyy;
  // face Jacobians: x-faces (constant x) and y-faces
  double JFx, JFy;
  double cfl_scaled;
};

// Device scalars of one context (time step, accumulated time, reduction slot, flags).
struct DevScalars {
  double dt;                   // current step
  double time;                 // accumulated time
  unsigned long long umax;     // max wave speed as ordered bits (non-negative doubles)
  unsigned int flags;          // bit 0: NaN wave speed / dt, bit 1: dt < 1e-14
  unsigned int blocks_done;    // CTAs of a wave-speed reduction that have added their maximum
  double dt_fixed;             // fixed step (> 0) or 0 for the CFL step
};

enum { FLAG_NONFINITE = 1u, FLAG_DT_SMALL = 2u, FLAG_TIMEOUT = 4u };

// Programmatic dependent launch (a kernel launched with programmatic stream serialization may be
// scheduled before its predecessor in the stream has finished): pdl_wait blocks until the
// predecessor grid has completed and its memory is visible (at once when the launch was not
// programmatic), so it comes before a kernel's first access to global data; pdl_trigger lets the
// next kernel's CTAs be scheduled as this one's finish.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// What an earlier launch wrote, read in a kernel that waits for it.  Not with __ldg (which const __restrict__ pointers
// can become too): ld.global.nc is for data that nobody writes while the kernel lives, and a kernel that
// waits lives beside the one that writes.  ld_dep is a plain load that stays behind the wait, and in order with
// the other such loads.  ld_after is one that may be scheduled freely (1 us per 512 x 256 step), through a pointer
// that after_wait has made a result of the wait, so that it cannot move above it either.
__device__ __forceinline__ double ld_dep(const double* p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ unsigned ld_dep(const unsigned* p) {
  unsigned v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
template <class T>
__device__ __forceinline__ T* after_wait(T* p) {
  asm volatile("" : "+l"(p));
  return p;
}
__device__ __forceinline__ double ld_after(const double* p) {
  double v;
  asm("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}

// the row of tiles of a CTA (tile_grid, launch.h)
__device__ __forceinline__ int tile_row() { return blockIdx.z * gridDim.y + blockIdx.y; }

// minmod of two arguments (limiting_kernels.cu:1470-1486): the smaller in magnitude when their signs
// agree, else 0.  Signs are compared as bits (a zero argument gives 0 either way).
__device__ __forceinline__ double minmod2(double a, double b) {
  const double m = fabs(a) < fabs(b) ? a : b;
  return (__double2hiint(a) ^ __double2hiint(b)) < 0 ? 0.0 : m;
}
// The same where an argument may be a NaN, which has no sign: against another number it gives 0, so that an element
// beside one with a NaN keeps its mean; 0 or NaN against a NaN gives NaN.
__device__ __forceinline__ double minmod2_nan(double a, double b) {
  if (!(fabs(a) < fabs(b)) && !(fabs(a) >= fabs(b))) return b != b && !(fabs(a) > 0.0) ? b : 0.0;
  return minmod2(a, b);
}
// Whether one of two values is infinite or a NaN, on the integer pipe.  The limiters test the cell sums of the two
// neighbours, which no infinity or NaN among their nodes leaves finite, once per slice and take minmod2_nan
// then.  p = 2, 512 x 256: 33.2 us per stage, 33.6 with the test in every minmod, 32.7 without; p = 3, 1024 x 512:
// 315, 329 and 305.
__device__ __forceinline__ bool nonfinite2(double a, double b) {
  return max((unsigned)__double2hiint(a) << 1, (unsigned)__double2hiint(b) << 1) >= 0xffe00000u;
}
template <bool NANS>
__device__ __forceinline__ double minmod2_of(double a, double b) {
  return NANS ? minmod2_nan(a, b) : minmod2(a, b);
}

// ---- hierarchical reconstruction of one 1D slice -------------------------------------------------
// Nodes are equispaced on [-1, 1]; a[n] are scaled Taylor coefficients, u(x) = sum a_n x^n / n!.  The
// limiter (limit_monomial, limiting_kernels.cu:1534-1583) compares, for k = P-1 .. 0, the cell means of
// the k-th derivative in the cell and its two neighbours, after taking from each the mean of the
// already limited higher terms.  So a cell enters only through the means of its derivatives 0 .. P-1 --
// P numbers, simple sums of its nodal values -- and the integrals over the neighbours' intervals
// are the constants 13/6 and 5/3.  Written out per order this is a quarter of the multiplications of the
// general form with its transform and integral tables.
// D: the P means times fixed factors (P = 1: 2 u; P = 2: 6 u, 2 u'; P = 3: 8 u, 2 u', 8/9 u'').
template <int P>
__device__ __forceinline__ void hr_moments(const double* v, double* D) {
  if constexpr (P == 1) {
    D[0] = v[0] + v[1];
  } else if constexpr (P == 2) {
    D[0] = (v[0] + v[2]) + 4.0 * v[1];
    D[1] = v[2] - v[0];
  } else {
    const double s0 = v[0] + v[3], s1 = v[1] + v[2];
    D[0] = s0 + 3.0 * s1;
    D[1] = v[3] - v[0];
    D[2] = s0 - s1;
  }
}
// The cell mean of the nodal values v.  P = 2: from the middle node, so that the mean of a constant is that constant --
// as 1/6 of D[0] it drifts by the rounding of 1/6 with every pass (2.7e-15 of the state after 20 steps of a 64 x 32
// bubble, 6e-16 this way).
template <int P>
__device__ __forceinline__ double hr_mean(const double* v) {
  if constexpr (P == 1) return 0.5 * (v[0] + v[1]);
  if constexpr (P == 2) return v[1] + ((v[0] + v[2]) - 2.0 * v[1]) * (1.0 / 6.0);
  if constexpr (P == 3) return 0.125 * ((v[0] + v[3]) + 3.0 * (v[1] + v[2]));
}
// the limited Taylor coefficients of the cell with nodal values v and moments DC between neighbours DL and DR
template <int P, bool NANS>
__device__ __forceinline__ void hr_limit_of(const double* DL, const double* DC, const double* DR, const double* v,
                                            double* lim) {
  if constexpr (P == 1) {
    lim[1] = 0.25 * minmod2_of<NANS>(DC[0] - DL[0], DR[0] - DC[0]);
    lim[0] = 0.5 * DC[0];
  } else if constexpr (P == 2) {
    lim[2] = 0.25 * minmod2_of<NANS>(DC[1] - DL[1], DR[1] - DC[1]);
    lim[1] = minmod2_of<NANS>((DC[0] - DL[0]) * (1.0 / 12.0) + lim[2], (DR[0] - DC[0]) * (1.0 / 12.0) - lim[2]);
    lim[0] = v[1] + (((v[0] + v[2]) - 2.0 * v[1]) - lim[2]) * (1.0 / 6.0);
  } else {
    lim[3] = 0.5625 * minmod2_of<NANS>(DC[2] - DL[2], DR[2] - DC[2]);
    lim[2] = minmod2_of<NANS>(0.25 * (DC[1] - DL[1]) + lim[3], 0.25 * (DR[1] - DC[1]) - lim[3]);
    const double t = lim[3] * (-5.0 / 6.0);
    lim[1] = minmod2_of<NANS>(0.0625 * (DC[0] - DL[0]) + (t + lim[2]), 0.0625 * (DR[0] - DC[0]) + (t - lim[2]));
    lim[0] = 0.125 * DC[0] - lim[2] * (1.0 / 6.0);
  }
}
template <int P>
__device__ __forceinline__ void hr_limit(const double* DL, const double* DC, const double* DR, const double* v,
                                         double* lim) {
  if (nonfinite2(DL[0], DR[0])) hr_limit_of<P, true>(DL, DC, DR, v, lim);
  else hr_limit_of<P, false>(DL, DC, DR, v, lim);
}
// the cell mean kept, the rest zero (average_monomial, limiting_kernels.cu:1777-1790)
template <int P>
__device__ __forceinline__ void hr_flat(const double* v, double* lim) {
  lim[0] = hr_mean<P>(v);
#pragma unroll
  for (int m = 1; m <= P; ++m) lim[m] = 0.0;
}
// nodal values -> scaled Taylor coefficients, and back
template <int P>
__device__ __forceinline__ void to_mono(const double* v, double* a) {
  if constexpr (P == 1) {
    a[0] = 0.5 * (v[0] + v[1]);
    a[1] = 0.5 * (v[1] - v[0]);
  } else if constexpr (P == 2) {
    a[0] = v[1];
    a[1] = 0.5 * (v[2] - v[0]);
    a[2] = (v[0] + v[2]) - 2.0 * v[1];
  } else {
    const double s0 = v[0] + v[3], s1 = v[1] + v[2], d0 = v[3] - v[0], d1 = v[2] - v[1];
    a[0] = 0.0625 * (9.0 * s1 - s0);
    a[1] = 0.0625 * (27.0 * d1 - d0);
    a[2] = 1.125 * (s0 - s1);
    a[3] = 3.375 * (d0 - 3.0 * d1);
  }
}
template <int P>
__device__ __forceinline__ void to_lag(const double* a, double* v) {
  if constexpr (P == 1) {
    v[0] = a[0] - a[1];
    v[1] = a[0] + a[1];
  } else if constexpr (P == 2) {
    const double e = a[0] + 0.5 * a[2];
    v[0] = e - a[1];
    v[1] = a[0];
    v[2] = e + a[1];
  } else {
    const double e1 = a[0] + 0.5 * a[2], o1 = a[1] + a[3] * (1.0 / 6.0);
    const double e3 = a[0] + a[2] * (1.0 / 18.0), o3 = a[1] * (1.0 / 3.0) + a[3] * (1.0 / 162.0);
    v[0] = e1 - o1;
    v[1] = e3 - o3;
    v[2] = e3 + o3;
    v[3] = e1 + o1;
  }
}
// E of a slice from its limited pressure and alpha and its kinetic energy: coefficients m >= 1 are those
// of rho e + K, rho e the Leibniz product of p and alpha (internal_energy_multifluid,
// limiting_kernels.cu:160-199), and the cell mean of E is kept (reconstruct_energy, :111-156)
template <int P>
__device__ __forceinline__ void hr_energy(const double* plim, const double* alim, const double* Kmono, double mean,
                                          double* E) {
  E[1] = (plim[1] * alim[0] + plim[0] * alim[1]) + Kmono[1];
  if constexpr (P >= 2) E[2] = (plim[2] * alim[0] + (2.0 * plim[1] * alim[1] + plim[0] * alim[2])) + Kmono[2];
  if constexpr (P >= 3)
    E[3] = (plim[3] * alim[0] + (3.0 * (plim[2] * alim[1] + plim[1] * alim[2]) + plim[0] * alim[3])) + Kmono[3];
  E[0] = P >= 2 ? mean - E[P >= 2 ? 2 : 0] * (1.0 / 6.0) : mean;
}

// The same as a form that the kernels are written over.  NM moments of a slice are what its neighbours need.
template <int P>
struct HrSums {
  static constexpr int NM = P;
  static __device__ __forceinline__ void moments(const double* v, double* D) { hr_moments<P>(v, D); }
  static __device__ __forceinline__ void limit(const double* DL, const double* DC, const double* DR, const double* v,
                                               double* lim) {
    hr_limit<P>(DL, DC, DR, v, lim);
  }
  static __device__ __forceinline__ void flat(const double*, const double* v, double* lim) { hr_flat<P>(v, lim); }
  static __device__ __forceinline__ void mono(const double* v, double* a) { to_mono<P>(v, a); }
  static __device__ __forceinline__ void lag(const double* a, double* v) { to_lag<P>(a, v); }
  // E rebuilt from the limited coefficients of p and alpha, the limited kinetic energy K and the slice
  // vE of E before (nodal values, and out)
  static __device__ __forceinline__ void energy(const double* plim, const double* alim, const double* K, const double* vE,
                                                double* E) {
    double Km[P + 1], El[P + 1];
    to_mono<P>(K, Km);
    hr_energy<P>(plim, alim, Km, hr_mean<P>(vE), El);
    to_lag<P>(El, E);
  }
  static __device__ __forceinline__ double rcp(double x);  // physics.cuh
};

// Cubic elements in 2D.  There the limited scheme itself multiplies a difference of rounding by 10 to 15 per
// step, up to some 4e-8 of the state (with any flux; p <= 2, 1D and the unlimited scheme leave it at 1e-15), so
// after five steps a run repeats an earlier one to 1e-11 only if every sum keeps its terms, their order and
// their rounding.  This form does: a slice's Taylor coefficients are formed with a transform that carries
// the rounding of its numerical inversion (within 1e-14 of 9/16, 27/16, 9/8, 27/8, ...),
// reciprocals are correctly rounded, and the kernels apply the operations in the order written here.
// (in constant memory: as literals they would be moved into registers)
static __constant__ double c_hr3_T[4][4] = {
    {-0x1.000000000000cp-4, 0x1.2p-1, 0x1.2p-1, -0x1.ffffffffffff6p-5},
    {0x1.0000000000006p-4, -0x1.afffffffffffdp+0, 0x1.b000000000002p+0, -0x1.fffffffffffebp-5},
    {0x1.2000000000001p+0, -0x1.2000000000001p+0, -0x1.2000000000003p+0, 0x1.1ffffffffffffp+0},
    {-0x1.bp+1, 0x1.43ffffffffffep+3, -0x1.4400000000002p+3, 0x1.afffffffffffep+1}};
static __constant__ double c_hr3_Ti[4][4] = {
    {0x1.0000000000007p+0, -0x1.0000000000001p+0, 0x1.ffffffffffffep-2, -0x1.5555555555557p-3},
    {0x1.0000000000003p+0, -0x1.5555555555559p-2, 0x1.c71c71c71c72p-5, -0x1.948b0fcd6ea03p-8},
    {0x1.ffffffffffffcp-1, 0x1.5555555555553p-2, 0x1.c71c71c71c71cp-5, 0x1.948b0fcd6e9bdp-8},
    {0x1.0000000000001p+0, 0x1.0000000000001p+0, 0x1p-1, 0x1.5555555555556p-3}};
struct HrTab3 {
  static constexpr int NM = 3;
  static __device__ __forceinline__ void mono(const double* v, double* a) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      double s = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) s += c_hr3_T[m][i] * v[i];
      a[m] = s;
    }
  }
  static __device__ __forceinline__ void lag(const double* a, double* v) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      double s = 0;
#pragma unroll
      for (int m = 0; m < 4; ++m) s += c_hr3_Ti[i][m] * a[m];
      v[i] = s;
    }
  }
  // D: the integrals of u, u' and u'' over the cell (integrate_monomial_derivative(_bounds),
  // limiting_kernels.cu:1748-1775), from the Taylor coefficients
  static __device__ __forceinline__ void means(const double* a, double* D) {
    D[0] = __fma_rn(a[2], 2.0 / 6.0, 2.0 * a[0]);
    D[1] = __fma_rn(a[3], 2.0 / 6.0, 2.0 * a[1]);
    D[2] = 2.0 * a[2];
  }
  static __device__ __forceinline__ void moments(const double* v, double* D) {
    double a[4];
    mono(v, a);
    means(a, D);
  }
  template <bool NANS>
  static __device__ __forceinline__ void limit_of(const double* DL, const double* DC, const double* DR, double* lim) {
    // a neighbour's mean less that of the limited higher terms over its interval, [-3, -1] or [1, 3]
    auto side = [](double d, double r) { return 0.5 * __dsub_rn(d, r); };
    auto pick = [](double l, double c, double r) { return minmod2_of<NANS>(0.5 * __dsub_rn(c, l), 0.5 * __dsub_rn(r, c)); };
    lim[3] = pick(0.5 * DL[2], 0.5 * DC[2], 0.5 * DR[2]);
    const double r3 = __dmul_rn(lim[3], 26.0 / 6.0);
    lim[2] = pick(side(DL[1], r3), side(DC[1], __dmul_rn(lim[3], 2.0 / 6.0)), side(DR[1], r3));
    const double r2 = __dmul_rn(lim[2], 26.0 / 6.0);
    lim[0] = side(DC[0], __dmul_rn(lim[2], 2.0 / 6.0));
    lim[1] = pick(side(DL[0], __fma_rn(lim[3], -80.0 / 24.0, r2)), lim[0], side(DR[0], __fma_rn(lim[3], 80.0 / 24.0, r2)));
  }
  static __device__ __forceinline__ void limit(const double* DL, const double* DC, const double* DR, const double*,
                                               double* lim) {
    if (nonfinite2(DL[0], DR[0])) limit_of<true>(DL, DC, DR, lim);
    else limit_of<false>(DL, DC, DR, lim);
  }
  static __device__ __forceinline__ void flat(const double* DC, const double*, double* lim) {
    lim[0] = 0.5 * DC[0];
    lim[1] = lim[2] = lim[3] = 0.0;
  }
  static __device__ __forceinline__ void energy(const double* plim, const double* alim, const double* K, const double* vE,
                                                double* E) {
    constexpr double binom[4][4] = {{1, 0, 0, 0}, {1, 1, 0, 0}, {1, 2, 1, 0}, {1, 3, 3, 1}};
    double Km[4], Em[4], El[4], re[4];
    mono(K, Km);
    mono(vE, Em);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      double s = 0;
#pragma unroll
      for (int k = 0; k <= m; ++k) s += binom[m][k] * plim[m - k] * alim[k];
      re[m] = s;
    }
#pragma unroll
    for (int m = 1; m < 4; ++m) El[m] = re[m] + Km[m];
    El[0] = Em[0] - (1.0 / 6.0) * (El[2] - Em[2]);
    lag(El, E);
  }
  static __device__ __forceinline__ double rcp(double x) { return __drcp_rn(x); }
};
// the form of the 2D limiters
template <int P>
using Hr2 = std::conditional_t<P == 3, HrTab3, HrSums<P>>;

}  // namespace dgb
