"""The work a user of this solver has it do, as cases that can be run, timed and checked.

A case is one call sequence on a problem that the program keeps: set a state, advance it a few steps, read
the state back (device buffers in the reference layout, or pinned host memory), or the same for an
ensemble of problems advanced together.  `exact` restates the scheme in plain float64 torch.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

import dg_b200 as dgb
from dg_b200 import _ffi, learned

DEV = "cuda"
SCHEMES = {"ssprk3": dgb.SSPRK3, "rk4": dgb.RK4}
STAGES = {"ssprk3": 3, "rk4": 4}


def _run(dim, order, nx, ny, flux, limiter, scheme, steps, ic, form="fp64", learned=False, n_mass=0, host=False):
    return {"kind": "run", "dim": dim, "order": order, "nx": nx, "ny": ny, "flux": flux, "limiter": limiter,
            "scheme": scheme, "steps": steps, "ic": ic, "form": form, "learned": learned, "n_mass": n_mass, "host": host}


def listed():
    return [
        # the 1D two-fluid shock tube of the decks: 12,000 DOF, every launch counts
        dict(_run(1, 2, 1000, 1, "roe", "m2l", "rk4", 25, "tube"), name="tube_p2_1000"),
        # a fine 1D chain of uneven length at the highest order
        dict(_run(1, 3, 19997, 1, "hll", "m2l", "ssprk3", 25, "tube"), name="tube_p3_19997"),
        # a coarse 2D study, a few thousand elements: parameter scans, tests, first looks
        dict(_run(2, 2, 64, 32, "rusanov", "m2l", "ssprk3", 20, "bubble"), name="bubble_p2_64x32"),
        # the shock-bubble workload the benchmark is quoted on
        dict(_run(2, 2, 512, 256, "rusanov", "m2l", "ssprk3", 8, "bubble"), name="bubble_p2_512x256"),
        # the same from host memory: upload, advance between two outputs, download
        dict(_run(2, 2, 512, 256, "rusanov", "m2l", "ssprk3", 8, "bubble", host=True), name="bubble_p2_host"),
        # a grid of odd extents, the reference's own integrator and flux
        dict(_run(2, 2, 501, 251, "roe", "hrl", "rk4", 5, "quadrants"), name="ragged_p2_501x251"),
        # linear elements on a larger grid, without a limiter on a smooth flow
        dict(_run(2, 1, 1000, 500, "rusanov", "none", "rk4", 6, "smooth"), name="smooth_p1_1000x500"),
        # cubic elements, Roe flux: the largest single problem
        dict(_run(2, 3, 1024, 512, "roe", "m2l", "ssprk3", 4, "bubble"), name="bubble_p3_1024x512"),
        # a passive mass fraction marks the bubble
        dict(_run(2, 2, 512, 256, "rusanov", "m2l", "ssprk3", 5, "bubble", n_mass=1), name="marked_p2_512x256"),
        # the mixed FP32/FP64 form on the four-quadrant problem
        dict(_run(2, 2, 768, 768, "rusanov", "m2l", "ssprk3", 5, "quadrants", form="mixed"), name="mixed_p2_768x768"),
        # mixed form with the learned indicator gating the limiter, scored every eighth step
        dict(_run(2, 2, 768, 768, "rusanov", "m2l", "ssprk3", 8, "quadrants", form="mixed", learned=True),
             name="learned_p2_768x768"),
        # an ensemble of uneven 1D and 2D problems advanced together
        {"name": "ensemble_24_8", "kind": "ensemble", "n1d": 24, "n2d": 8, "mix": 1, "steps": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: sizes over their logarithm, odd ones among them."""
    what = rng.choice(["1d", "1d", "2d", "2d", "2d", "2d", "host", "marked", "mixed", "learned", "ensemble"])
    if what == "ensemble":
        return {"kind": "ensemble", "n1d": rng.randint(4, 32), "n2d": rng.randint(1, 8), "mix": rng.randint(2, 10 ** 6),
                "steps": rng.randint(2, 4)}
    scheme = rng.choice(["ssprk3", "rk4"])
    limiter = rng.choice(["m2l", "m2l", "hrl"])
    if what == "1d":
        flux = rng.choice(["rusanov", "hll", "roe"])  # HLL, whose momentum row is the reference's, needs m2l here
        return _run(1, rng.randint(1, 3), _log(rng, 200, 20000), 1, flux, "m2l" if flux == "hll" else limiter, scheme,
                    rng.randint(10, 25), "tube")
    if what == "mixed" or what == "learned":
        nx, ny = 2 * _log(rng, 64, 384), _log(rng, 128, 768)
        order = 2 if what == "learned" else rng.randint(1, 3)
        if order == 3:
            ny = (ny + 1) // 2
        return _run(2, order, nx, ny, rng.choice(["rusanov", "roe"]), "m2l" if what == "learned" else limiter,
                    "ssprk3", rng.randint(3, 8) if what == "mixed" else 8, "quadrants", "mixed", what == "learned")
    if what == "marked":
        return _run(2, rng.randint(1, 2), 2 * _log(rng, 32, 256), _log(rng, 32, 256), rng.choice(["rusanov", "roe"]),
                    limiter, scheme, rng.randint(2, 4), "bubble", n_mass=rng.randint(1, 3))
    ic = rng.choice(["bubble", "quadrants", "smooth"])
    if ic == "smooth" and rng.random() < 0.5:
        limiter = "none"
    if what == "host":
        return _run(2, rng.randint(1, 3), _log(rng, 64, 400), _log(rng, 32, 200), rng.choice(["rusanov", "roe"]), limiter,
                    scheme, rng.randint(2, 8), ic, host=True)
    order = rng.randint(1, 3)
    most = {1: 900, 2: 700, 3: 480}[order]
    return _run(2, order, _log(rng, 33, most), _log(rng, 16, most), rng.choice(["rusanov", "roe"]), limiter, scheme,
                rng.randint(3, 6), ic)


# ---- inputs ---------------------------------------------------------------------------------------


def _gmsh_nodes(dim, p):
    """(ix, iy) of each node of a Gmsh line / quadrangle of order p, lattice indices ascending."""
    if dim == 1:
        return [(0, 0), (p, 0)] + [(i, 0) for i in range(1, p)]
    if p == 0:
        return [(0, 0)]
    out = [(0, 0), (p, 0), (p, p), (0, p)]
    out += [(i, 0) for i in range(1, p)] + [(p, i) for i in range(1, p)]
    out += [(p - i, p) for i in range(1, p)] + [(0, p - i) for i in range(1, p)]
    if p >= 2:
        out += [(i + 1, j + 1) for i, j in _gmsh_nodes(2, p - 2)]
    return out


DOMAIN = {"tube": (0.0, 1.0, 0.0, 1.0), "bubble": (0.0, 2.0, 0.0, 1.0), "quadrants": (0.0, 1.0, 0.0, 1.0),
          "smooth": (0.0, 1.0, 0.0, 1.0)}
# sides in the order bottom, right, top, left (1D: left, right)
SIDES = {"tube": ("transmissive", "reflective", "transmissive", "transmissive"),
         "bubble": ("reflective", "transmissive", "reflective", "transmissive"),
         "quadrants": ("transmissive",) * 4, "smooth": ("periodic",) * 4}


@functools.lru_cache(maxsize=16)
def _mesh_problem(dim, order, nx, ny, flux, limiter, ic, n_mass):
    """The problem of a mesh (host only), which a program keeps from one state to the next."""
    x0, x1, y0, y1 = DOMAIN[ic]
    return dgb.Problem.structured(dim, order, nx, ny, x0, x1, y0, y1, SIDES[ic], flux=flux, limiter=limiter,
                                  cfl=0.4 if dim == 1 else 0.3, n_mass=n_mass)


def _initial(c, seed):
    """Seeded state [element, field, node] on the GPU.  Jumps sit on element faces."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)
    rnd = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    x0, x1, y0, y1 = DOMAIN[c["ic"]]
    p, nx, ny = c["order"], c["nx"], c["ny"]
    lat = torch.tensor(_gmsh_nodes(c["dim"], p), device=DEV, dtype=torch.float64) / p
    ex = torch.arange(nx, device=DEV, dtype=torch.float64)
    hx = (x1 - x0) / nx
    if c["dim"] == 1:
        x = x0 + hx * (ex[:, None] + lat[None, :, 0])
        left = (x0 + hx * (ex + 0.5) < 0.5)[:, None].expand_as(x)
        rho = torch.where(left, 1.0, 0.125) + 1e-3 * (2 * rnd(*x.shape) - 1)
        u = torch.zeros_like(x)
        pr = torch.where(left, 1.0, 0.1) * (1 + 0.1 * rnd(1))
        gam = torch.where(left, 1.4, 1.6).double()
        al = 1 / (gam - 1)
        return torch.stack([rho, rho * u, al * pr + 0.5 * rho * u * u, al], 1).contiguous()
    hy = (y1 - y0) / ny
    ey = torch.arange(ny, device=DEV, dtype=torch.float64)
    ex, ey = ex.repeat(ny), ey.repeat_interleave(nx)
    x, y = x0 + hx * (ex[:, None] + lat[None, :, 0]), y0 + hy * (ey[:, None] + lat[None, :, 1])
    cx, cy = (x0 + hx * (ex + 0.5))[:, None], (y0 + hy * (ey + 0.5))[:, None]
    ph = 2 * math.pi * rnd(6)
    wave = torch.sin(2 * math.pi * x + ph[0]) * torch.sin(2 * math.pi * y + ph[1])
    if c["ic"] == "smooth":
        rho, u, v = 1 + 0.2 * wave, 1 + 0.0 * x, 1 + 0.0 * x
        pr = 1 + 0.02 * torch.sin(2 * math.pi * (x + y) + ph[2])
        gam, mark = 1.4 + 0.2 * torch.sin(2 * math.pi * x + ph[3]) * torch.sin(2 * math.pi * y + ph[4]), 0.0 * x
    elif c["ic"] == "bubble":
        th = torch.atan2(cy - 0.5, cx - 0.5)
        amp, r = 0.002 * (2 * rnd(6) - 1), 0.2 + 0 * cx
        for k in range(6):
            r = r + amp[k] * torch.cos((k + 2) * th + ph[k])
        shock, inside = cx < 0.2, (cx - 0.5) ** 2 + (cy - 0.5) ** 2 < r * r
        pick = lambda s, b, o: torch.where(shock, s, torch.where(inside, b, o)).double().expand_as(x)  # noqa: E731
        # Mach-1.5 shock in air (gamma 1.4, rho 1, p 1) into a bubble of gamma 1.67, rho 0.138
        rho = pick(1.8620689655172413, 0.138, 1.0) * (1 + 0.01 * wave)
        u, v, pr, gam = pick(0.8216, 0.0, 0.0), 0.0 * x, pick(2.4583333333333335, 1.0, 1.0), pick(1.4, 1.67, 1.4)
        mark = pick(0.0, 1.0, 0.0)
    else:
        q = (cx >= 0.5).long() + 2 * (cy >= 0.5).long()
        r0, p0 = 0.1 + 1.9 * rnd(4), 0.1 + 1.9 * rnd(4)
        rho, pr = r0[q].expand_as(x) * (1 + 0.01 * wave), p0[q].expand_as(x)
        u, v = (2 * rnd(4) - 1)[q].expand_as(x), (2 * rnd(4) - 1)[q].expand_as(x)
        gam, mark = torch.where(rnd(4) < 0.5, 1.4, 1.67).double()[q].expand_as(x), (q % 2).double().expand_as(x)
    al = 1 / (gam - 1)
    f = [rho, rho * u, rho * v, al * pr + 0.5 * rho * (u * u + v * v), al]
    f += [rho * (mark if k % 2 == 0 else 1 - mark) for k in range(c["n_mass"])]
    return torch.stack(f, 1).contiguous()


def _members(c):
    """The problems of an ensemble: 1D chains and 2D grids whose extents are multiples of 64."""
    r = random.Random(c["mix"])
    out = [_run(1, r.randint(1, 3), _log(r, 200, 20000), 1, "rusanov", "m2l", "ssprk3", c["steps"], "tube")
           for _ in range(c["n1d"])]
    return out + [_run(2, 2, 64 * r.randint(1, 4), 64 * r.randint(1, 4), "rusanov", "m2l", "ssprk3", c["steps"],
                       "quadrants") for _ in range(c["n2d"])]


def _solver(c):
    return dgb.DGSolver(_mesh_problem(c["dim"], c["order"], c["nx"], c["ny"], c["flux"], c["limiter"], c["ic"],
                                      c["n_mass"]), device=torch.cuda.current_device())


def prepare(case, seed):
    if case["kind"] == "ensemble":
        cs = _members(case)
        U = [_initial(c, 1000 * seed + k) for k, c in enumerate(cs)]
        solvers = [_solver(c) for c in cs]
        state = {"case": case, "solvers": solvers, "batch": dgb.DGBatch(solvers), "U": U,
                 "out": [torch.empty_like(u) for u in U]}
        torch.cuda.synchronize()
        return state
    s = _solver(case)
    if case["form"] != "fp64":
        s.set_form(case["form"])
    if case["learned"]:
        learned.set_indicator(s, learned.load()[0], every=8)
    U = _initial(case, seed)
    if case["host"]:
        host, out = U.cpu().pin_memory(), torch.empty(U.shape, dtype=torch.float64).pin_memory()
        return {"case": case, "solver": s, "U": host.view(-1).numpy(), "out": out.view(-1).numpy(), "keep": (host, out)}
    state = {"case": case, "solver": s, "U": U, "out": torch.empty_like(U)}
    torch.cuda.synchronize()  # the solver works on a stream of its own
    return state


# ---- the call ---------------------------------------------------------------------------------------


def run(state):
    c, L = state["case"], _ffi.lib()
    if c["kind"] == "ensemble":
        for s, u in zip(state["solvers"], state["U"]):
            _ffi.check(L.dgb_set_state_device(s._h, u.data_ptr()))
        state["batch"].advance(c["steps"])
        for s, o in zip(state["solvers"], state["out"]):
            _ffi.check(L.dgb_get_state_device(s._h, o.data_ptr()))
        return {"U": state["out"], "time": state["batch"].case_stats()[0]}
    s = state["solver"]
    if c["host"]:
        s.set_state(state["U"])
        t = s.advance(c["steps"], 0.0, scheme=SCHEMES[c["scheme"]])
        return {"U": s.get_state(state["out"]), "time": t}
    _ffi.check(L.dgb_set_state_device(s._h, state["U"].data_ptr()))
    t = s.advance(c["steps"], 0.0, scheme=SCHEMES[c["scheme"]])
    _ffi.check(L.dgb_get_state_device(s._h, state["out"].data_ptr()))
    return {"U": state["out"], "time": t}


def work(case):
    """Per step and DOF: each stage reads its input (and the step's base state) and writes its output once
    (SSP-RK3 8 doubles, RK4 20), the CFL step reads the state once; plus the state in and out.  Flops: the
    sum-factorised contractions, the point fluxes and Riemann solvers, the limiter's transforms."""
    b = f = 0.0
    for c in _members(case) if case["kind"] == "ensemble" else [case]:
        n1, d, nf = c["order"] + 1, c["dim"], c["dim"] + 3 + c["n_mass"]
        ne, ns = c["nx"] * c["ny"], (c["order"] + 1) ** c["dim"]
        dof, st = ne * ns * nf, STAGES[c["scheme"]]
        b += dof * 8.0 * (c["steps"] * (8 if st == 3 else 20) + 1 + 4)
        q = n1 if d == 1 else (2 if n1 == 2 else n1 + 1)
        if d == 1:
            per = 2 * nf * n1 * (2 * q + n1) + 40 * q + 150 + (0 if c["limiter"] == "none" else 2 * nf * n1 * (4 * n1))
        else:
            per = 2 * nf * (2 * (q * n1 * n1 + q * q * n1) + 3 * n1 * n1) + 40 * q * q + 2 * n1 * 150
            per += 0 if c["limiter"] == "none" else 2 * 2 * (nf + 1) * n1 * n1 * (4 * n1)
        f += per * float(ne) * st * c["steps"]
    return {"bytes": b, "flops": f}


def tolerance(case):
    # FP64 against the same scheme in plain float64 torch: 2e-16 to 5e-15 in the 2-norm, 2e-12 where the
    # mesh spacing that the step is formed from carries the rounding of its coordinates.  Mixed form (FP32
    # contractions on FP64 anchors): 6e-9 to 2e-8, at most 8e-7 at a node.  Learned, against the same run
    # with FP64 contractions: 2e-8 to 1.4e-7 and 1.3e-6 (a cell whose score sits at the threshold may be
    # limited or not).
    if case["kind"] == "run" and case["learned"]:
        return {"rel": 6e-7, "max": 5e-6}
    if case["kind"] == "run" and case["form"] == "mixed":
        return {"rel": 8e-8, "max": 3e-6}
    return {"rel": 1e-11, "max": 1e-9}


# ---- the scheme in plain float64 torch ----------------------------------------------------------------


def _tables(p, ng):
    xs = np.linspace(-1.0, 1.0, p + 1)
    xq, wq = np.polynomial.legendre.leggauss(ng)
    xf, wf = np.polynomial.legendre.leggauss(p + 1)
    V = np.vander(xs, p + 1, increasing=True)
    C = np.linalg.inv(V)  # column i: the power coefficients of l_i
    ev = lambda x: np.vander(x, p + 1, increasing=True) @ C  # noqa: E731
    dv = lambda x: np.stack([n * x ** max(n - 1, 0) for n in range(p + 1)], 1) @ C  # noqa: E731
    xm, wm = np.polynomial.legendre.leggauss(p + 2)
    M = (ev(xm).T * wm) @ ev(xm)
    fact = np.array([math.factorial(n) for n in range(p + 1)], float)
    Ti = V / fact  # scaled Taylor coefficients -> nodal values
    mom = lambda a, b: np.array([[0.0 if n < k else (b ** (n - k + 1) - a ** (n - k + 1)) / math.factorial(n - k + 1)  # noqa: E731
                                  for n in range(p + 1)] for k in range(p + 1)])
    t = lambda a: torch.tensor(np.ascontiguousarray(a), device=DEV)  # noqa: E731
    return {"B": t(ev(xq)), "D": t(dv(xq)), "w": t(wq), "Bf": t(ev(xf)), "wf": t(wf), "Mi": t(np.linalg.inv(M)),
            "T": t(np.linalg.inv(Ti)), "Ti": t(Ti), "C": mom(-1, 1), "L": mom(-3, -1), "R": mom(1, 3)}


def _riemann(flux, L, R, n, d, ny):
    """Interface flux and the non-conservative term; n: the normal's components; fields first."""
    rl, rr, El, Er, al, ar = L[0], R[0], L[d + 1], R[d + 1], L[d + 2], R[d + 2]
    vl, vr = [L[1 + k] / rl for k in range(d)], [R[1 + k] / rr for k in range(d)]
    unl, unr = sum(v * m for v, m in zip(vl, n)), sum(v * m for v, m in zip(vr, n))
    pl, pr = (El - 0.5 * rl * sum(v * v for v in vl)) / al, (Er - 0.5 * rr * sum(v * v for v in vr)) / ar
    cl, cr = torch.sqrt((1 + 1 / al) * pl / rl), torch.sqrt((1 + 1 / ar) * pr / rr)
    fl = [rl * unl] + [rl * unl * v + pl * m for v, m in zip(vl, n)] + [(El + pl) * unl]
    fr = [rr * unr] + [rr * unr * v + pr * m for v, m in zip(vr, n)] + [(Er + pr) * unr]
    ul, ur = [rl] + L[1:d + 1] + [El], [rr] + R[1:d + 1] + [Er]
    Yl, Yr = L[d + 3:], R[d + 3:]
    if flux == "rusanov":
        s = torch.maximum(unl.abs() + cl, unr.abs() + cr)
        F = [0.5 * (a + b - s * (y - x)) for a, b, x, y in zip(fl, fr, ul, ur)] + [-0.5 * s * (ar - al)]
        F += [0.5 * (x * unl + y * unr) - s * (y - x) for x, y in zip(Yl, Yr)]
        return F, -0.25 * (unl + unr) * (ar - al)
    if flux == "hll":  # 1D; the momentum jump is taken in the velocities
        sl, sr = torch.minimum(unl - cl, unr - cr), torch.maximum(unl + cl, unr + cr)
        iw = 1 / (sr - sl).abs()
        ul, ur = [rl, vl[0], El], [rr, vr[0], Er]
        mid = [(sr * a - sl * b + sl * sr * (y - x)) * iw for a, b, x, y in zip(fl, fr, ul, ur)]
        va = -0.5 * (unl + unr).abs() * (al - ar)
        mid.append(sl * sr * (ar - al) * iw - 0.5 * (sr + sl).abs() * iw * va)
        left, right = fl + [-0.5 * va], fr + [0.5 * va]
        z = torch.zeros_like(rl)
        F = [torch.where(sl > 0, a, torch.where((sl < 0) & (sr > 0), m, torch.where(sr < 0, b, z)))
             for a, m, b in zip(left, mid, right)]
        return F, 0.25 * (unl + unr) * (al - ar)
    t = (-n[1], n[0]) if d == 2 else ()
    rt = torch.sqrt(rr / rl)
    avg = lambda x, y: (x + rt * y) / (1 + rt)  # noqa: E731
    rho, v, H = rt * rl, [avg(x, y) for x, y in zip(vl, vr)], avg((El + pl) / rl, (Er + pr) / rr)
    un, al_, i = sum(a * m for a, m in zip(v, n)), avg(al, ar), avg(pl * al, pr * ar)
    g1 = 1 / al_
    c = torch.sqrt(g1 * (H - 0.5 * sum(a * a for a in v)))
    dp = g1 * g1 * (al_ * (pr * ar - pl * al) - i * (ar - al))
    w0, w3 = (dp - rho * c * (unr - unl)) / (2 * c * c), (dp + rho * c * (unr - unl)) / (2 * c * c)
    w2 = rr - rl - dp / (c * c)
    a0, a1, a3 = (un - c).abs(), un.abs(), (un + c).abs()
    k0, k2, k3, k4 = a0 * w0, a1 * w2, a3 * w3, a1 * (ar - al)
    D = [k0 + k2 + k3] + [k0 * (x - c * m) + k2 * x + k3 * (x + c * m) for x, m in zip(v, n)]
    D.append(k0 * (H - un * c) + k2 * 0.5 * sum(a * a for a in v) + k3 * (H + un * c) + k4 * g1 * i)
    if d == 2:
        ut = sum(a * m for a, m in zip(v, t))
        k1 = a1 * rho * sum((y - x) * m for x, y, m in zip(vl, vr, t)) / c
        D[1], D[2], D[3] = D[1] + k1 * c * t[0], D[2] + k1 * c * t[1], D[3] + k1 * ut * c
    F = [0.5 * (a + b) - 0.5 * x for a, b, x in zip(fl, fr, D)] + [-0.5 * k4]
    for x, y in zip(Yl, Yr):
        Y = avg(x / rl, y / rr)
        F.append(0.5 * (x * unl + y * unr) - 0.5 * ((k0 + k2 + k3) * Y + a1 * (y - x - (w0 + w2 + w3) * Y)))
    return F, -0.5 * un * (ar - al)


class _Scheme:
    """u[field, iy, ix, y, x] (1D: one node and element in y), nodes ascending."""

    def __init__(self, c):
        self.c, self.d, p = c, c["dim"], c["order"]
        x0, x1, y0, y1 = DOMAIN[c["ic"]]
        self.h = ((x1 - x0) / c["nx"], (y1 - y0) / c["ny"])
        self.t = _tables(p, p + 1 if self.d == 1 or p == 1 else p + 2)
        s = SIDES[c["ic"]]
        self.side = ((s[0], s[1]),) if self.d == 1 else ((s[3], s[1]), (s[0], s[2]))
        self.dx = self.h[0] if self.d == 1 else min(self.h)
        self.cfl = (0.4 if self.d == 1 else 0.3) * self.dx / (2 * p + 1)

    def pressure(self, u):
        d = self.d
        return (u[d + 1] - 0.5 * sum(u[1 + k] ** 2 for k in range(d)) / u[0]) / u[d + 2]

    def dt(self, u):
        d = self.d
        a = torch.sqrt((1 + 1 / u[d + 2]) * self.pressure(u) / u[0])
        return self.cfl / float((torch.stack([(u[1 + k] / u[0]).abs() for k in range(d)]).amax(0) + a).max())

    def faces(self, u, ax):
        """Face fluxes across axis ax (0: x, 1: y): F and nc per face, faces 0 .. n along the axis."""
        d, nodes, elems = self.d, u.ndim - 3 - ax, u.ndim - 1 - ax
        lo, hi = u.select(nodes, 0), u.select(nodes, u.shape[nodes] - 1)  # first / last node of every element
        if d == 2:
            lo, hi = torch.einsum("gj,fjyx->fgyx", self.t["Bf"], lo), torch.einsum("gj,fjyx->fgyx", self.t["Bf"], hi)
        e = elems - 1
        n = lo.shape[e]
        first, last = lo.narrow(e, 0, 1), hi.narrow(e, n - 1, 1)
        sgn = torch.ones([1 if k != e - 1 else n + 1 for k in range(lo.ndim - 1)], device=DEV, dtype=torch.float64)
        mirror = lambda q, kind: torch.stack([-f if kind == "reflective" and k == 1 + ax else f for k, f in enumerate(q)])  # noqa: E731
        if self.side[ax][0] == "periodic":
            L, R = torch.cat([last, hi], e), torch.cat([lo, first], e)
        else:  # at a wall the inside state is L with its outward normal
            L = torch.cat([first, hi], e)
            R = torch.cat([mirror(first, self.side[ax][0]), lo.narrow(e, 1, n - 1), mirror(last, self.side[ax][1])], e)
            sgn.select(e - 1, 0).fill_(-1.0)
        z = torch.zeros_like(sgn)
        F, nc = _riemann(self.c["flux"], list(L), list(R), [sgn if k == ax else z for k in range(d)], d, 0)
        return torch.stack([sgn * f for f in F]), nc

    def du(self, u, dt):
        """dt M^-1 (volume, source and face terms)."""
        d, t = self.d, self.t
        B, D, w = t["B"], t["D"], t["w"]
        # 1D: the y direction is one node, one point of weight one
        By, Dy, wy = (B, D, w) if d == 2 else (torch.ones(1, 1, device=DEV, dtype=torch.float64),) * 2 + (torch.ones(1, device=DEV, dtype=torch.float64),)
        con = lambda a, b, q: torch.einsum("hj,fjgyx->fhgyx", a, torch.einsum("gi,fjiyx->fjgyx", b, q))  # noqa: E731
        back = lambda a, b, q: torch.einsum("hj,fhiyx->fjiyx", a, torch.einsum("gi,fhgyx->fhiyx", b, q))  # noqa: E731
        ug = con(By, B, u)
        W = (wy[:, None] * w[None, :])[None, :, :, None, None]
        m = (2 / self.h[0], 2 / self.h[1])
        J = self.h[0] / 2 * (self.h[1] / 2 if d == 2 else 1.0)
        p, v = self.pressure(ug), [ug[1 + k] / ug[0] for k in range(d)]
        r = torch.zeros_like(u)
        src = 0
        for ax in range(d):
            f = torch.stack([ug[1 + ax]] + [ug[1 + k] * v[ax] + (p if k == ax else 0) for k in range(d)] +
                            [(ug[d + 1] + p) * v[ax], torch.zeros_like(p)] + [y * v[ax] for y in ug[d + 3:]])
            f = W * (J * m[ax]) * f
            r += back(By, D, f) if ax == 0 else back(Dy, B, f)
            src = src - v[ax] * m[ax] * (con(By, D, u[d + 2:d + 3]) if ax == 0 else con(Dy, B, u[d + 2:d + 3]))[0]
        r[d + 2] += back(By, B, (W[0] * J * src)[None])[0]
        for ax in range(d):
            F, nc = self.faces(u, ax)
            e, n = F.ndim - 1 - ax, u.shape[u.ndim - 1 - ax]
            one = torch.zeros(u.shape[0], *[1] * (F.ndim - 1), device=DEV, dtype=torch.float64)
            one[d + 2] = 1.0
            qr, ql = (F + one * nc).narrow(e, 0, n), (-F + one * nc).narrow(e, 1, n)
            if d == 2:
                k = 0.5 * self.h[1 - ax]
                qr, ql = (torch.einsum("gj,fgyx->fjyx", k * t["wf"][:, None] * t["Bf"], q) for q in (qr, ql))
            nodes = u.ndim - 3 - ax
            r.select(nodes, 0).add_(qr)
            r.select(nodes, u.shape[nodes] - 1).add_(ql)
        r = torch.einsum("ki,fjiyx->fjkyx", t["Mi"], r)
        return (dt / J) * (torch.einsum("kj,fjiyx->fkiyx", t["Mi"], r) if d == 2 else r)

    def limit_axis(self, q, ax, keep):
        """Hierarchical reconstruction along an axis of the scaled Taylor coefficients q (nodes of the
        axis first); keep: leave the coefficients at a reflective wall."""
        t, n1 = self.t, q.shape[0]
        e = q.ndim - 1 - ax
        lo, hi = torch.roll(q, 1, e), torch.roll(q, -1, e)
        lim = [None] * n1
        for m in range(n1 - 1, 0, -1):
            avg = []
            for a, tab in ((lo, "L"), (q, "C"), (hi, "R")):
                s = sum(a[n] * t["C"][m - 1][n] for n in range(m - 1, n1))
                s = s - sum((lim[n] * t[tab][m - 1][n] for n in range(m + 1, n1)), torch.zeros_like(s))
                avg.append(0.5 * s)
            c1, c2 = 0.5 * (avg[1] - avg[0]), 0.5 * (avg[2] - avg[1])
            lim[m] = torch.where(torch.sign(c1) == torch.sign(c2), torch.sign(c1) * torch.minimum(c1.abs(), c2.abs()), 0.0)
            center = avg[1]
        lim[0] = center
        out = torch.stack(lim)
        for k, kind in enumerate(self.side[ax]):
            if kind == "periodic":
                continue
            at = 0 if k == 0 else q.shape[e] - 1
            cell = q.select(e, at)
            flat = torch.zeros_like(cell)
            flat[0] = 0.5 * sum(cell[n] * t["C"][0][n] for n in range(n1))
            out.select(e, at).copy_(cell if keep and kind == "reflective" else flat)
        return out

    def limit_pass(self, q, E, ax, names):
        """One direction: quantities q[k] and, under m2l, the energy E rebuilt from p and alpha."""
        nodes = 1 - ax
        T, Ti = self.t["T"], self.t["Ti"]
        mono = lambda x: torch.tensordot(T, x, dims=([1], [nodes]))  # noqa: E731 (coefficient axis first)
        lag = lambda x: torch.movedim(torch.tensordot(Ti, x, dims=([1], [0])), 0, nodes)  # noqa: E731
        lim = []
        for k, x in enumerate(q):
            lim.append(self.limit_axis(mono(x), ax, E is None and names[k] == 1 + ax))
        out = [lag(x) for x in lim]
        if E is None:
            return torch.stack(out), None
        d = self.d
        K = mono(0.5 * sum(out[1 + k] ** 2 for k in range(d)) / out[0])
        a, p, Em = lim[d + 1], lim[d + 2], mono(E)
        n1 = a.shape[0]
        El = [None] + [sum(math.comb(m, k) * p[m - k] * a[k] for k in range(m + 1)) + K[m] for m in range(1, n1)]
        El[0] = Em[0] - sum((El[k] - Em[k]) / math.factorial(k + 1) for k in range(2, n1, 2))
        return torch.stack(out), lag(torch.stack(El))

    def limit(self, u):
        d, kind = self.d, self.c["limiter"]
        if kind == "none":
            return u
        if kind == "hrl":
            for ax in range(d):
                u = self.limit_pass(u, None, ax, list(range(u.shape[0])))[0]
            return u
        q = torch.stack([u[k] for k in range(d + 1)] + [u[d + 2], self.pressure(u)] + [y for y in u[d + 3:]])
        E = u[d + 1]
        for ax in range(d):
            q, E = self.limit_pass(q, E, ax, None)
        return torch.stack([q[k] for k in range(d + 1)] + [E, q[d + 1]] + [y for y in q[d + 3:]])

    def advance(self, u, steps):
        time = 0.0
        for _ in range(steps):
            dt = self.dt(u)
            time += dt
            if self.c["scheme"] == "ssprk3":
                a = self.limit(u + self.du(u, dt))
                a = self.limit(0.75 * u + 0.25 * (a + self.du(a, dt)))
                u = self.limit(u / 3 + 2 / 3 * (a + self.du(a, dt)))
            else:
                acc, x = u, u
                for k, (gam, beta) in enumerate(zip((1 / 6, 1 / 3, 1 / 3, 1 / 6), (0.5, 0.5, 1.0, 0.0))):
                    du = self.du(x, dt)
                    acc = acc + gam * du
                    if k < 3:
                        x = self.limit(u + beta * du)
                u = self.limit(acc)
        return u, time


def _exact_run(c, seed):
    n1, d = c["order"] + 1, c["dim"]
    U = _initial(c, seed)
    at = [ix + n1 * iy for ix, iy in _gmsh_nodes(d, c["order"])]
    inv = [at.index(k) for k in range(len(at))]
    u = U[:, :, inv].permute(1, 2, 0).reshape(U.shape[1], n1 if d == 2 else 1, n1, c["ny"], c["nx"])
    u, time = _Scheme(c).advance(u, c["steps"])
    return u.reshape(U.shape[1], len(at), -1).permute(2, 0, 1)[:, :, at].contiguous(), time


def exact(case, seed):
    if case["kind"] == "ensemble":
        got = [_exact_run(c, 1000 * seed + k) for k, c in enumerate(_members(case))]
        return {"U": [u for u, _ in got], "time": np.array([t for _, t in got])}
    if case["learned"]:
        return None  # which cells are limited is the network's decision
    u, time = _exact_run(case, seed)
    return {"U": u.reshape(-1).cpu().numpy() if case["host"] else u, "time": time}
