"""Limited runs of cubic elements in 2D repeat their recorded states.

The limited scheme at p = 3 multiplies differences of rounding by 10 to 15 per step (p <= 2, 1D and unlimited
runs do not), so that kernels whose sums have other terms or another order are off by 1e-10 after a dozen
steps, although each of them is as close to the scheme as the other.  The kernels of such runs therefore keep
terms, order and rounding (device/tile2d_ordered.cuh, HrTab3).  The states were recorded with the
one-thread-per-element kernels they stem from (commit 94dfbfa), every 29th value.  The bound: one rounding of
1e-16 that differs reaches 1e-11 to 1e-10 in these runs, so 1e-13 tells a kernel that repeats them from any
other; grids with elements outside the 32 x 2 blocks, both fluxes, limiters and schemes."""
from pathlib import Path

import numpy as np
import pytest

import dg_b200 as dgb

pytestmark = pytest.mark.gpu

RECORDED = Path(__file__).parent / "recorded" / "cubic_limited.npz"


def initial(prob, nx, ny):
    """Four quadrants with a density bump, by basic operations only (the same bits on any host)."""
    t = np.arange(16)
    ex, ey = np.arange(nx * ny) % nx, np.arange(nx * ny) // nx
    x, y = (ex[:, None] + (t % 4) / 3) / nx, (ey[:, None] + (t // 4) / 3) / ny
    q = ((2 * ex >= nx) + 2 * (2 * ey >= ny))[:, None] + 0 * t
    rho, u, v, p, al = (np.array(w)[q] for w in ([1.0, 0.4, 0.8, 1.5], [0.3, -0.4, 0.6, 0.1], [-0.2, 0.5, 0.3, -0.7],
                                                [1.0, 0.5, 0.7, 1.3], [2.5, 1.5, 2.5, 1.5]))
    rho = rho * (1 + 0.02 / (1 + 30 * (x - 0.3) * (x - 0.3) + 20 * (y - 0.6) * (y - 0.6)))
    U = np.empty((nx * ny, 5, 16))
    U[:, :, prob.array("tensor_perm")] = np.stack([rho, rho * u, rho * v, al * p + 0.5 * rho * (u * u + v * v), al], 1)
    return U.ravel()


@pytest.mark.parametrize("run", ["72x41_roe_hrl_ssprk3_12", "64x48_rusanov_m2l_ssprk3_16", "72x41_rusanov_hrl_rk4_16"])
def test_recorded_states(run):
    size, flux, limiter, scheme, steps = run.split("_")
    nx, ny = map(int, size.split("x"))
    prob = dgb.Problem.structured(2, 3, nx, ny, 0.0, 1.0, 0.0, 1.0, ("transmissive",) * 4, flux=flux, limiter=limiter,
                                  cfl=0.3)
    s = dgb.DGSolver(prob)
    s.set_state(initial(prob, nx, ny))
    s.advance(int(steps), 0.0, scheme=getattr(dgb, scheme.upper()))
    U, want = s.get_state()[::29], np.load(RECORDED)[run]
    s.close()
    assert np.linalg.norm(U - want) <= 1e-13 * np.linalg.norm(want)


def test_solve_without_accumulator():
    """dgb_solve has neither a stage base nor an accumulator: DU = dt M^-1 R of the residual entry."""
    prob = dgb.Problem.structured(2, 3, 34, 5, flux="rusanov", limiter="m2l", cfl=0.3)
    U = initial(prob, 34, 5)
    s = dgb.DGSolver(prob)
    DU, R = s.solve(1e-3, U).reshape(-1, 16), s.dg_solver(U).reshape(-1, 16)
    Minv = prob.array("Minv")[:256].reshape(16, 16)  # symmetric
    s.close()
    want = 1e-3 * R @ Minv
    assert np.abs(DU - want).max() <= 1e-12 * np.abs(want).max()
