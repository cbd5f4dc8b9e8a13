"""Grids with more rows of tiles than a launch has in grid.y (65,535): the residual's and the limiter's rows of
tiles go on in grid.z.  Against the generic kernels (DGB_NO_TILE=1): the same sums in another order, one step,
so within 1e-12 of the state's scale (some 100 products per value and stage, each 1e-16)."""
import numpy as np
import pytest

import dg_b200 as dgb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,ny,limiter,scheme", [(2, 140001, "none", dgb.SSPRK3), (1, 530001, "m2l", dgb.RK4)])
def test_narrow_tall_grid(monkeypatch, order, ny, limiter, scheme):
    prob = dgb.Problem.structured(2, order, 2, ny, 0.0, 0.2, 0.0, 0.1 * ny, ("reflective", "transmissive") * 2, flux="rusanov",
                                  limiter=limiter, cfl=0.3)
    U = prob.init_state("quadrants", seed=3).reshape(2 * ny, 5, -1)
    U[:, 0] *= 1 + 0.01 * np.random.default_rng(ny).random(U[:, 0].shape)
    out = []
    for generic in (False, True):
        if generic:
            monkeypatch.setenv("DGB_NO_TILE", "1")
        s = dgb.DGSolver(prob)
        s.set_state(U.ravel())
        s.advance(1, 1e-3, scheme=scheme)
        out.append(s.get_state())
        s.close()
    assert np.isfinite(out[1]).all() and np.abs(out[1] - U.ravel()).max() > 1e-3
    assert np.abs(out[0] - out[1]).max() <= 1e-12 * np.abs(out[1]).max()
