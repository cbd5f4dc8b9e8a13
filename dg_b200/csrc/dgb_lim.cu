// The one-launch 2D limiter of structured grids (lim2d_kernel, device/limiter2d_tile.cuh): dispatch
// over order, method and mass fractions, and its launches.
#include <cuda_runtime.h>

#include "../../include/dgb.h"
#include "device/limiter2d_tile.cuh"
#include "launch.h"

namespace dgb {

namespace {

template <int P, int METHOD, int NY>
int launch_lim(dgb_ctx* c, const double* in, double* out) {
  using Dm = LimDims<P, METHOD, NY>;
  auto k = lim2d_kernel<P, METHOD, NY>;
  DGB_CUDA(allow_dynamic_smem(k, Dm::smem_bytes));
  const dim3 grid = tile_grid((c->nx + 29) / 30, (c->ny + Dm::ROWS - 1) / Dm::ROWS), block(32, Dm::N1, Dm::ROWS + 2);
  ProfScope ps(c, KC_LIMITER);
  DGB_CUDA(launch_pdl(c, k, grid, block, Dm::smem_bytes, LimArgs{c->ld, c->ne}, c->nx, c->ny, in, (const int*)c->nbr, out,
                      (const DevScalars*)c->scal));
  return 0;
}

template <int NY>
int dispatch_lim(dgb_ctx* c, const double* in, double* out) {
  switch (c->p * 10 + c->limiter) {
    case 11: return launch_lim<1, 1, NY>(c, in, out);
    case 12: return launch_lim<1, 2, NY>(c, in, out);
    case 21: return launch_lim<2, 1, NY>(c, in, out);
    case 22: return launch_lim<2, 2, NY>(c, in, out);
    case 31: return launch_lim<3, 1, NY>(c, in, out);
    case 32: return launch_lim<3, 2, NY>(c, in, out);
    default: return set_error(DGB_ERR_UNSUPPORTED, "limiter not available on the device path");
  }
}

}  // namespace

// hrl / m2l from `in` into `out` (in != out); contexts with lim_out only
int limit2d_out(dgb_ctx* c, const double* in, double* out) {
  switch (c->nmass) {
    case 0: return dispatch_lim<0>(c, in, out);
    case 1: return dispatch_lim<1>(c, in, out);
    case 2: return dispatch_lim<2>(c, in, out);
    case 3: return dispatch_lim<3>(c, in, out);
    default: return set_error(DGB_ERR_UNSUPPORTED, "limiter not available on the device path");
  }
}

}  // namespace dgb
