"""The mixed form is the caller's permission to use FP32 contractions; FP64 kernels are the faster ones, so both
forms run FP64 kernels: the same launches and the same bits, but for limited cubic elements, whose FP64 form
keeps the order of its sums (test_gpu_cubic.py) and whose mixed form does not.  There the scheme amplifies the
rounding differences to some 4e-8 of the state: within 1e-6 per field in L1 after 30 steps.
"""
import numpy as np
import pytest

from conftest import perturbed_state

pytestmark = pytest.mark.gpu
WALLS = ("reflective", "transmissive", "reflective", "transmissive")


def per_field(a, b, info, norm="max"):
    """Per-field error of a against b; the two momentum components are scaled together (by the
    momentum magnitude), since one of them is nearly zero in these flows."""
    A = np.asarray(a).reshape(info.n_elem, info.n_fields, info.n_s)
    B = np.asarray(b).reshape(info.n_elem, info.n_fields, info.n_s)
    red = (lambda x: np.abs(x).max()) if norm == "max" else (lambda x: np.abs(x).sum())
    out = []
    for f in range(info.n_fields):
        scale = red(B[:, f]) if f not in (1, 2) else max(red(B[:, 1]), red(B[:, 2]))
        out.append(float(red(A[:, f] - B[:, f]) / scale))
    return out


@pytest.mark.parametrize("flux,order,limiter,nx,ny", [
    ("rusanov", 2, "m2l", 128, 64), ("roe", 2, "hrl", 100, 46), ("rusanov", 1, "m2l", 64, 33), ("roe", 3, "none", 64, 32)])
def test_forms_give_the_same_bits(flux, order, limiter, nx, ny):
    import dg_b200 as dgb
    prob = dgb.Problem.structured(2, order, nx, ny, 0.0, 2.0, 0.0, 1.0, WALLS, flux=flux, limiter=limiter, cfl=0.3)
    U0 = prob.init_state("quadrants" if limiter == "none" else "shock_bubble", seed=7)
    out = []
    for form in ("fp64", "mixed"):
        s = dgb.DGSolver(prob)
        s.set_form(form)
        U = s.limit(U0)
        f = s.dg_solver(U)
        s.set_state(U)
        t = s.advance(2, 1e-5, scheme=dgb.SSPRK3) if limiter == "none" else s.advance(20, 0.0, scheme=dgb.SSPRK3)
        out.append((f, s.get_state(), t))
        s.close()
    assert np.isfinite(out[0][1]).all()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("flux", ["rusanov", "roe"])
def test_cubic_residuals_agree(flux):
    import dg_b200 as dgb
    prob = dgb.Problem.structured(2, 3, 64, 32, 0.0, 2.0, 0.0, 1.0, WALLS, flux=flux, limiter="m2l", cfl=0.3)
    s = dgb.DGSolver(prob)
    U0 = s.limit(perturbed_state(prob, "shock_bubble", 5))
    f64, d64 = s.dg_solver(U0), s.solve(1e-3, U0)
    s.set_form("mixed")
    err = per_field(s.dg_solver(U0), f64, prob.info) + per_field(s.solve(1e-3, U0), d64, prob.info)
    s.close()
    assert max(err) < 1e-12, err  # the same sums of some 100 products in another order


def test_mixed_steps_close_to_fp64_p3_roe():
    """The 2048 x 1024 p=3 Roe configuration's form at a smaller size: 30 steps, per-field L1 and
    Linf against the FP64 form, and the drift of the conserved totals."""
    import dg_b200 as dgb
    prob = dgb.Problem.structured(2, 3, 128, 64, 0.0, 2.0, 0.0, 1.0, WALLS, flux="roe", limiter="m2l", cfl=0.3)
    ref = dgb.DGSolver(prob)
    mix = dgb.DGSolver(prob)
    try:
        U0 = ref.limit(prob.init_state("shock_bubble", seed=7))
        mix.set_form("mixed")
        tot = {}
        for name, s in (("fp64", ref), ("mixed", mix)):
            s.set_state(U0)
            c0 = s.conservation()
            s.advance(30, 0.0, scheme=dgb.SSPRK3)
            tot[name] = (c0, s.conservation())
        l1 = per_field(mix.get_state(), ref.get_state(), prob.info, norm="l1")
        li = per_field(mix.get_state(), ref.get_state(), prob.info, norm="max")
        print("p=3 Roe mixed vs FP64 after 30 steps, per-field relative L1:", l1, "Linf:", li)
        assert max(l1) < 1e-6 and max(li) < 1e-4
        # the conserved totals (which change through the open boundaries) of the two forms agree
        for name, (c0, c1) in tot.items():
            print(name, "conserved totals before/after:", c0, c1)
        c0, r1, m1 = tot["fp64"][0], tot["fp64"][1], tot["mixed"][1]
        scale = np.abs(c0).copy()
        scale[1:3] = np.abs(c0[:3]).max()  # momentum totals start near zero: mass scale
        assert np.all(np.abs(m1 - r1) <= 1e-7 * scale)
    finally:
        ref.close()
        mix.close()


def test_mixed_form_rejected_where_not_built():
    import dg_b200 as dgb
    prob = dgb.Problem.structured(2, 3, 41, 32, flux="roe", limiter="m2l")  # odd nx: no tiled kernel
    s = dgb.DGSolver(prob)
    try:
        with pytest.raises(dgb.DGBError):
            s.set_form("mixed")
    finally:
        s.close()
