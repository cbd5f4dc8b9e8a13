"""Runs of many steps: dgb_advance replays several captured steps at a time once a context has run some (five
per graph after a hundred steps).  The same kernels in the same order, so the states, the times and the
launch counts are those of single steps bit for bit, whatever the remainder."""
import numpy as np
import pytest

import dg_b200 as dgb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,scheme", [(1, dgb.RK4), (1, dgb.SSPRK3), (2, dgb.RK4), (2, dgb.SSPRK3)])
@pytest.mark.parametrize("dt", [0.0, 1e-4])
def test_long_runs_equal_single_steps(dim, scheme, dt):
    prob = (dgb.Problem.structured(1, 2, 130, 1, flux="roe", limiter="m2l", cfl=0.4) if dim == 1 else
            dgb.Problem.structured(2, 2, 20, 12, flux="rusanov", limiter="m2l", cfl=0.3))
    U0 = prob.init_state("riemann" if dim == 1 else "quadrants", seed=5)
    long_, short = dgb.DGSolver(prob), dgb.DGSolver(prob)
    for s in (long_, short):
        s.set_state(U0)
    t = 0.0
    for n in (96, 10, 13, 9):  # single steps, then graphs of five with remainders 0 and 3, then single ones
        t_long = long_.advance(n, dt, scheme=scheme)
        launches = long_.last_timing()[1]
        t_short = 0.0
        for _ in range(n):
            t_short += short.advance(1, dt, scheme=scheme)
        assert launches == n * short.last_timing()[1]
        assert abs(t_long - t_short) <= 1e-14 * n * abs(t_short)  # one sum of n steps against n sums
        assert np.array_equal(long_.get_state(), short.get_state())
    long_.close()
    short.close()
