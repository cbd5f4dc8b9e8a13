"""The tiled 2D residual (one thread per element and quadrature column) against the generic kernels
(DGB_NO_TILE=1, any element order) on grids that cut its tiles: one element wide, one row high, odd
extents, extents just below and above the tile.  Both are the same sums in another order: a residual is
some 100 products per node, so they agree within 100 eps of the largest term; the bound is 1e-12 of
the largest residual, and 1e-11 of the state's scale after two steps with the limiter."""
import numpy as np
import pytest

import dg_b200 as dgb

pytestmark = pytest.mark.gpu

WALLS = ("reflective", "transmissive", "reflective", "transmissive")
OPEN = ("transmissive",) * 4
SIDES = ("transmissive", "reflective", "transmissive", "reflective")
PERIODIC = ("periodic",) * 4


def both(monkeypatch, order, nx, ny, bc, flux, limiter, scheme):
    out = []
    for generic in (False, True):
        if generic:
            monkeypatch.setenv("DGB_NO_TILE", "1")
        prob = dgb.Problem.structured(2, order, nx, ny, 0.0, 0.1 * nx, 0.0, 0.13 * ny, bc, flux=flux,
                                      limiter=limiter, cfl=0.3)
        rng = np.random.default_rng(order + 10 * nx + 1000 * ny)
        U = prob.init_state("quadrants", seed=nx + ny).reshape(nx * ny, 5, -1)
        U[:, 0] *= 1 + 0.01 * rng.random(U[:, 0].shape)
        s = dgb.DGSolver(prob)
        f = s.dg_solver(U.ravel())
        s.set_state(U.ravel())
        s.advance(2, 1e-4, scheme=scheme)
        out.append((f, s.get_state()))
        s.close()
        monkeypatch.delenv("DGB_NO_TILE", raising=False)
    return out


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("nx,ny,bc,flux,limiter,scheme", [
    (2, 2, OPEN, "roe", "none", dgb.SSPRK3),
    (5, 3, WALLS, "rusanov", "m2l", dgb.RK4),
    (17, 1, OPEN, "rusanov", "none", dgb.SSPRK3),
    (16, 4, PERIODIC, "rusanov", "hrl", dgb.RK4),
    (15, 5, SIDES, "roe", "m2l", dgb.SSPRK3),
    (18, 3, WALLS, "roe", "hrl", dgb.RK4),
    (33, 9, PERIODIC, "roe", "m2l", dgb.SSPRK3),
    (64, 7, SIDES, "rusanov", "m2l", dgb.RK4),
])
def test_cut_tiles(monkeypatch, order, nx, ny, bc, flux, limiter, scheme):
    (f0, u0), (f1, u1) = both(monkeypatch, order, nx, ny, bc, flux, limiter, scheme)
    assert np.isfinite(f0).all() and np.isfinite(u0).all()
    assert np.abs(f0 - f1).max() <= 1e-12 * np.abs(f1).max()
    assert np.abs(u0 - u1).max() <= 1e-11 * np.abs(u1).max()
