"""A NaN in one element and the limiter: the minmod of a NaN and another number is 0, so the elements beside it keep
their mean in that field and the rest is limited as without it (limiting_kernels.cu:1470-1486: a NaN has no sign)."""
import numpy as np
import pytest

import dg_b200 as dgb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("tiled", [True, False])
def test_nan_stays_in_its_element(monkeypatch, order, tiled):
    if not tiled:
        monkeypatch.setenv("DGB_NO_TILE", "1")
    nx, ny, n1 = 40, 11, order + 1
    rng = np.random.default_rng(order)
    for dim, e, step in ((1, 20, 1), (2, 4 * nx + 20, nx)):  # the direction limited last: x, y
        prob = dgb.Problem.structured(dim, order, nx, ny if dim == 2 else 1, flux="rusanov", limiter="hrl", cfl=0.3)
        U = np.zeros((prob.info.n_elem, prob.info.n_fields, prob.info.n_s))
        # every moment rises along x and y: none of its differences is 0
        t, perm = np.arange(n1 ** dim), prob.array("tensor_perm")
        rise = lambda a: np.cumsum(a + a * rng.random(nx))[np.arange(len(U)) % nx] + np.cumsum(a + a * rng.random(ny))[np.arange(len(U)) // nx]  # noqa: E731
        c = [rise(a)[:, None] for a in (0.5, 0.02, 0.02, 0.02)]
        U[:, :, perm] = sum(c[k] * ((t % n1) ** k + (t // n1) ** k) for k in range(4))[:, None, :]
        s = dgb.DGSolver(prob)
        clean = s.limit(U.ravel()).reshape(U.shape)
        bad = U.copy()
        bad[e, 0, perm] = np.nan
        got = s.limit(bad.ravel()).reshape(U.shape)
        s.close()
        assert np.isnan(got[e, 0]).all() and np.isfinite(np.delete(got[:, 0], [e], 0)).all()
        for k in (e - step, e + step):  # flat along that direction, and it was not without the NaN
            v, c = (u[k, 0, perm].reshape((n1,) * dim) for u in (got, clean))
            assert np.abs(v - v[:1]).max() <= 1e-13 * np.abs(v).max() < np.abs(c - c[:1]).max()
        touched = [19, 20, 21] if dim == 1 else [e + i + j * nx for i in (-1, 0, 1) for j in (-1, 0, 1)]
        far = np.delete(np.arange(len(U)), touched)
        assert np.array_equal(got[far, 0], clean[far, 0]) and np.array_equal(got[:, 1:], clean[:, 1:])
