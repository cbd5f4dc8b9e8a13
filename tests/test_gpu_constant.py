"""The limiter leaves a constant state as it is, bit for bit, however often it is applied: its mean is formed so that
no rounding of a constant factor enters (p = 3 in 2D carries the rounding of its transforms instead, HrTab3)."""
import numpy as np
import pytest

import dg_b200 as dgb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,order", [(1, 1), (1, 2), (1, 3), (2, 1), (2, 2)])
@pytest.mark.parametrize("limiter", ["hrl", "m2l"])
@pytest.mark.parametrize("tiled", [True, False])
def test_constant_state(monkeypatch, dim, order, limiter, tiled):
    if not tiled:
        monkeypatch.setenv("DGB_NO_TILE", "1")
    prob = dgb.Problem.structured(dim, order, 37, 11 if dim == 2 else 1, bc=("periodic",) * 4, flux="rusanov",
                                  limiter=limiter, cfl=0.3)
    field = [1.1, 0.3, 2.7, 1 / 0.67] if dim == 1 else [1.1, 0.3, -0.7, 2.7, 1 / 0.67]
    U0 = np.broadcast_to(np.array(field)[None, :, None], (prob.info.n_elem, len(field), prob.info.n_s)).ravel().copy()
    s = dgb.DGSolver(prob)
    U = U0
    for _ in range(20):
        U = s.limit(U)
    s.close()
    assert np.array_equal(U, U0)
