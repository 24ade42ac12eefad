"""Workloads of the solver, from one right-hand side of a few thousand cells to
3D grids of 17 million, through the entry points a program calls:

* ``run``     BlockSolver / cfd_set_state_device + run_device (cfd_run): CFL
              steps of a grid that lives on the device; the state comes back as
              the handle's own buffer, with every step's dt and log value;
* ``hostrun`` set_cons + run_device + cons: a small 1D program that keeps its
              arrays on the host;
* ``rhs``     cfd_rhs_noalloc: one right-hand side on the caller's buffers;
* ``hstep``   cfd_step_host: one CFL step of host code that keeps its state in
              pinned host memory;
* ``batch``   BlockBatch.run: independent Riemann problems of uneven grids;
* ``adjoint`` adjoint_record + adjoint_reverse: a gradient with checkpoints.

``exact`` restates the discretisation (characteristic reconstruction, HLLC or
Roe, the sixth-order midpoint-and-node difference, SSP-RK3) in plain torch.
"""
import ctypes as C
import math

import numpy as np
import torch

from cfd_inwsl_b200 import _lib, slabs, zone

DEV = "cuda:0"
G = 1.4
T_END = 1e3  # no output interval ends within a case
SCHEMES = {"wcns5": zone.InterMethod.WCNS5, "wenoz": zone.InterMethod.WCNSZ5, "teno": zone.InterMethod.TCNS5,
           "congz": zone.InterMethod.WCNS5CONGZ}
FLUXES = {"hllc": zone.FluxMethod.HLLC, "roe": zone.FluxMethod.ROE}


def _case(kind, flow, n, scheme, flux, form, bc, steps, cfl, **more):
    """n: cells per direction, comma separated; form: strict, fast (FP64) or mixed."""
    return dict(kind=kind, flow=flow, n=",".join(map(str, n)), scheme=scheme, flux=flux, form=form, bc=bc,
                steps=steps, cfl=cfl, **more)


def listed():
    """The 1D configuration (300 steps take it to about t = 0.16), one right-hand side for
    a caller with its own time stepper, the smallest vortex of the convergence
    study, the double Mach reflection with its wired boundaries, an odd 2D
    Riemann problem in the default flavour, the benchmark's vortex in the
    reference's roundings and a smaller one in the mixed form, Taylor-Green in
    the reference's roundings and, larger, in the default flavour, a batch of
    Riemann problems, a gradient at the adjoint configuration's size and a
    host-to-host step."""
    named = {
        "sod_400": _case("hostrun", "sod", (400,), "wcns5", "hllc", "strict", "outlet", 300, 0.5),
        "rhs_60x44": _case("rhs", "vortex", (60, 44), "wcns5", "hllc", "fast", "wrap", 1, 0.4),
        "vortex_64": _case("run", "vortex", (64, 64), "teno", "roe", "strict", "wrap", 24, 0.4),
        "double_mach_240x60": _case("run", "dmr", (240, 60), "teno", "hllc", "strict", "dmr", 24, 0.4),
        "riemann_301x203": _case("run", "riemann", (301, 203), "wcns5", "hllc", "fast", "outlet", 12, 0.5),
        "vortex_2048": _case("run", "vortex", (2048, 2048), "teno", "roe", "strict", "wrap", 3, 0.4),
        "vortex_1024_mixed": _case("run", "vortex", (1024, 1024), "teno", "roe", "mixed", "wrap", 6, 0.4),
        "tgv_128": _case("run", "tgv", (128, 128, 128), "wcns5", "hllc", "strict", "wrap", 3, 0.5),
        "tgv_256_fast": _case("run", "tgv", (256, 256, 256), "wcns5", "hllc", "fast", "wrap", 2, 0.5),
        "batch_24": _case("batch", "riemann", (128, 512), "wcns5", "hllc", "fast", "outlet", 6, 0.5, count=24),
        "adjoint_256": _case("adjoint", "density", (256, 256), "wcns5", "roe", "fast", "wrap", 40, 0.5, every=20),
        "host_step_2048x1000": _case("hstep", "vortex", (2048, 1000), "teno", "roe", "strict", "wrap", 1, 0.4),
    }
    return [dict(c, name=k) for k, c in named.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run1", "run2", "run2", "run2", "run3", "run3", "hostrun", "rhs", "batch", "adjoint", "hstep"])
    scheme = rng.choice(["wcns5", "wcns5", "teno", "teno", "wenoz", "congz"])
    flux = rng.choice(["hllc", "roe"])
    form = rng.choice(["strict", "fast", "mixed"])
    if kind in ("run1", "hostrun"):
        n = (_log_int(rng, 90, 6000),)
        one = "fast" if scheme == "wcns5" and form != "strict" else "strict"
        return _case("run" if kind == "run1" else kind, "sod", n, scheme, flux, one, "outlet",
                     rng.randint(20, 120), 0.5)
    # shocks and long runs in the default and mixed forms with the scheme they
    # are meant for: the others' cut-offs turn last-bit differences into larger
    # ones there, and such a user takes the strict form
    soft = scheme == "wcns5" or form == "strict"
    if kind == "run2":
        n = (_log_int(rng, 40, 1500), _log_int(rng, 40, 1500))
        steps = max(2, min(40, int(6e6 / (n[0] * n[1]))))
        flow = rng.random()
        if flow < 0.5:
            return _case("run", "vortex", n, scheme, flux, form, "wrap", steps if soft else min(steps, 4), 0.4)
        if flow < 0.65:
            k = _log_int(rng, 40, 200)
            return _case("run", "dmr", (4 * k, k), scheme, "hllc", "strict" if not soft else form, "dmr", 12, 0.4)
        return _case("run", "riemann", n, scheme, "hllc", form if soft else "strict", "outlet", steps, 0.5)
    if kind == "run3":
        n = tuple(_log_int(rng, 24, 200) for _ in range(3))
        steps = max(1, min(12 if soft else 3, int(6e6 / (n[0] * n[1] * n[2]))))
        return _case("run", "tgv", n, scheme, flux, form, "wrap", steps, 0.5)
    if kind == "rhs":
        n = (_log_int(rng, 40, 900), _log_int(rng, 40, 900))
        return _case("rhs", "vortex", n, scheme, flux, rng.choice(["strict", "fast"]), "wrap", 1, 0.4)
    if kind == "batch":
        return _case("batch", "riemann", (96, _log_int(rng, 128, 500)), scheme, "hllc", form if soft else "strict", "outlet",
                     rng.randint(3, 6), 0.5, count=_log_int(rng, 4, 32))
    if kind == "adjoint":
        n = (_log_int(rng, 64, 320), _log_int(rng, 64, 320))
        return _case("adjoint", "density", n, "wcns5", "roe", rng.choice(["strict", "fast"]), "wrap", rng.randint(10, 40), 0.5, every=rng.choice([10, 20]))
    n = (_log_int(rng, 200, 2048), _log_int(rng, 100, 1000))
    return _case("hstep", "vortex", n, scheme, flux, form, "wrap", 1, 0.4)


# ---------------------------------------------------------------- inputs
def _cells(case):
    return [int(x) for x in case["n"].split(",")]


def _gen(seed):
    return np.random.default_rng(seed)


def _extent(case):
    return {"vortex": 10.0, "tgv": 2 * math.pi, "dmr": 4.0}.get(case["flow"], 1.0)


def _cons(prim):
    """(rho, u.., p) -> conserved, both stacked along dim 0."""
    r, v, p = prim[0], prim[1:-1], prim[-1]
    return torch.cat([r[None], r * v, (p / (G - 1) + 0.5 * r * (v * v).sum(0))[None]])


def _initial(case, n, seed):
    """Conserved state (nvar, [nz,] [ny,] nx), FP64 on the device. Spacing is the
    x extent over n[0] in every direction, as Info.geth has it."""
    rng = _gen(seed)
    h = _extent(case) / n[0]
    x = [((torch.arange(k, device=DEV, dtype=torch.float64)) + 0.5) * h for k in n]
    flow = case["flow"]
    if flow == "sod":
        a = 1 + 0.1 * rng.uniform(-1, 1, 4)
        left = x[0] < 0.5
        rho = torch.where(left, torch.full_like(x[0], a[0]), 0.125 * a[1])
        p = torch.where(left, torch.full_like(x[0], a[2]), 0.1 * a[3])
        return _cons(torch.stack([rho, torch.zeros_like(rho), p]))
    if flow == "tgv":
        ph = rng.uniform(0, 0.5, 3)
        Z, Y, X = torch.meshgrid(x[2], x[1], x[0], indexing="ij")
        # whole waves along each extent, whatever its cell count
        X, Y, Z = (q * (n[0] / m) + s for q, m, s in ((X, n[0], ph[0]), (Y, n[1], ph[1]), (Z, n[2], ph[2])))
        u = torch.sin(X) * torch.cos(Y) * torch.cos(Z)
        v = -torch.cos(X) * torch.sin(Y) * torch.cos(Z)
        p = 100 / 1.4 + (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2) / 16
        # density along the isentrope, as the developed flow has it
        return _cons(torch.stack([(p * 1.4 / 100) ** (1 / G), u, v, torch.zeros_like(u), p]))
    Y, X = torch.meshgrid(x[1], x[0], indexing="ij")
    if flow == "vortex":
        beta, cx, cy = 5 + rng.uniform(-0.5, 0.5), 5 + rng.uniform(-1, 1), 5 + rng.uniform(-1, 1)
        # stretched to the box, so that it is smooth and periodic on any of them
        dx = torch.remainder(X - cx + 5.0, 10.0) - 5.0
        dy = torch.remainder(Y * (n[0] / n[1]) - cy + 5.0, 10.0) - 5.0
        r2 = dx * dx + dy * dy
        f = beta / (2 * math.pi) * torch.exp(0.5 * (1 - r2))
        T = 1 - (G - 1) * beta ** 2 / (8 * G * math.pi ** 2) * torch.exp(1 - r2)
        rho = T ** (1 / (G - 1))
        return _cons(torch.stack([rho, 1 - f * dy, 1 + f * dx, rho ** G]))
    if flow == "riemann":
        # the batched configuration's quadrants; the less dissipative schemes get weaker ones
        r0, p0, v = (0.1, 0.05, 1.0) if case["scheme"] == "wcns5" else (0.4, 0.4, 0.5)
        P = torch.tensor([[rng.uniform(r0, 2), rng.uniform(-v, v), rng.uniform(-v, v), rng.uniform(p0, 2)]
                          for _ in range(4)], device=DEV, dtype=torch.float64)
        q = (X >= 0.5).long() + 2 * (Y >= 0.5 * n[1] * h).long()
        return _cons(P[q].permute(2, 0, 1).contiguous())
    if flow == "dmr":
        post = _dmr_post()
        front = X < 1.0 / 6.0 + Y / math.sqrt(3.0)
        pre = [1.4, 0.0, 0.0, 1.0]
        prim = torch.stack([torch.where(front, torch.full_like(X, a), b) for a, b in zip(post, pre)])
        k = rng.uniform(1, 3, 2)
        prim[0] = prim[0] * (1 + 0.01 * torch.sin(2 * math.pi * k[0] * X) * torch.sin(2 * math.pi * k[1] * Y))
        return _cons(prim)
    # "density": a smooth periodic density field over a uniform flow
    rho = torch.ones_like(X)
    for _ in range(8):
        kx, ky = (int(k) for k in rng.integers(1, 5, 2))
        ph = rng.uniform(0, 2 * math.pi)
        rho = rho + 4e-3 * torch.sin(2 * math.pi * (kx * X + ky * Y / (n[1] * h)) + ph)
    one = torch.ones_like(X)
    return _cons(torch.stack([rho, 0.5 * one, 0.3 * one, one / G]))


def _dmr_post():
    return [8.0, 8.25 * math.cos(math.pi / 6), -8.25 * math.sin(math.pi / 6), 116.5]


def _info(case, n):
    info = zone.Info()
    info.iMax = [k + 1 for k in n] + [2] * (3 - len(n))
    info.dim = info.getDim()
    L = _extent(case)
    info.calZone = [0.0, L, 0.0, L, 0.0, L]
    info.nCase = 4 if case["flow"] == "dmr" else 0
    info.CFL = case["cfl"]
    info.interMethod = SCHEMES[case["scheme"]]
    info.fluxMethod = FLUXES[case["flux"]]
    info.strict = case["form"] == "strict"
    info.precision = int(case["form"] == "mixed")
    info.endStep = 1
    info.outputDt = T_END
    return info


def _solver(case, n):
    info = _info(case, n)
    return zone.BlockSolver(info, periodic=case["bc"] == "wrap")


def _sizes(case, seed):
    lo, hi = _cells(case)
    rng = _gen(1000)  # the grids belong to the case, the states to the seed
    return [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(case["count"])]


def _aos(u):
    return np.ascontiguousarray(u.reshape(u.shape[0], -1).t().cpu().numpy())


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sizes = _sizes(case, seed)
        batch = zone.BlockBatch([_info(case, (m, m)) for m in sizes], periodic=False)
        return {"case": case, "batch": batch, "sizes": sizes,
                "init": [_aos(_initial(case, (m, m), seed * 1000 + i)) for i, m in enumerate(sizes)]}
    n = _cells(case)
    s = _solver(case, n)
    u = _initial(case, n, seed)
    state = {"case": case, "solver": s, "n": n}
    if kind == "run":
        state["init"] = u.contiguous()
    elif kind == "hostrun":
        state["init"] = _aos(u)
    elif kind == "rhs":
        state |= {"u": u.contiguous(), "out": torch.empty_like(u)}
    elif kind == "hstep":
        state["in"] = torch.from_numpy(_aos(u)).pin_memory().numpy()
        state["out"] = torch.empty(state["in"].shape, dtype=torch.float64, pin_memory=True).numpy()
    else:  # adjoint
        state["init"] = _aos(u)
        state["grad"] = _gen(seed + 77).normal(size=state["init"].shape)
        state["dt"] = float(_adjoint_dt(case, n))
    return state


def _adjoint_dt(case, n):
    # sound speed about 1 beside (0.5, 0.3): the frozen step of the gradient study
    return case["cfl"] / ((1.0 + 0.5) * n[0] + (1.0 + 0.3) * n[0])


# ---------------------------------------------------------------- one pass
def _device_state(s):
    """The handle's current state as a tensor that shares its buffer."""
    ptr = C.c_void_p()
    _lib.check(s.lib.cfd_device_state(s.h, C.byref(ptr), None, None), s.h)
    view = slabs._DevArray(ptr.value, (s.nvar, *reversed(s.n[:s.dim])))
    view.owner = s  # the tensor holds the view, the view the handle that owns the buffer
    return torch.as_tensor(view, device=DEV)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        for i, info in enumerate(b.infos):
            info.t = 0.0
            b.set_cons(i, state["init"][i])
        t, steps = b.run(T_END, end_step=1, max_steps=case["steps"])
        return {"t": t, "steps": steps, "cons": [b.cons(i) for i in range(b.ncases)]}
    s = state["solver"]
    s.info.t = 0.0
    if kind == "run":
        _lib.check(s.lib.cfd_set_state_device(s.h, C.c_void_p(state["init"].data_ptr())), s.h)
        dts, linf = s.run_device(case["steps"])
        return {"dt": dts, "linf": linf, "state": _device_state(s)}
    if kind == "hostrun":
        s.set_cons(state["init"])
        dts, linf = s.run_device(case["steps"])
        return {"dt": dts, "linf": linf, "cons": s.cons, "t": s.info.t}
    if kind == "rhs":
        st = torch.cuda.current_stream().cuda_stream
        _lib.check(s.lib.cfd_rhs_noalloc(C.byref(s.cfg), C.c_void_p(state["u"].data_ptr()),
                                         C.c_void_p(state["out"].data_ptr()), 0.0, C.c_void_p(st)))
        return state["out"]
    if kind == "hstep":
        t, dt = C.c_double(0.0), C.c_double()
        _lib.check(s.lib.cfd_step_host(s.h, case["cfl"], T_END, _lib.ptr(state["in"]), _lib.ptr(state["out"]), C.byref(t),
                                       C.byref(dt)), s.h)
        return {"cons": state["out"], "t": t.value, "dt": dt.value}
    s.set_cons(state["init"])
    s.adjoint_record(state["dt"], case["steps"], case["every"])
    return {"gradient": s.adjoint_reverse(state["grad"]), "cons": s.cons}


# ---------------------------------------------------------------- what a pass needs
# FP64 operations of one face (its reconstruction, flux and difference) with
# each scheme's cheapest form, by dimension: 2 V interpolations of about 45
# (45 to 60 with three divisions), the projections and the Riemann flux
_FACE_FLOPS = {1: 560, 2: 830, 3: 1150}


def work(case):
    kind, steps = case["kind"], case["steps"]
    grids = [(m, m) for m in _sizes(case, 0)] if kind == "batch" else [_cells(case)]
    bytes_, flops = 0.0, 0.0
    for n in grids:
        d = len(n)
        cells = math.prod(n)
        state = 8 * cells * (d + 2)
        stages = 1 if kind == "rhs" else 3 * steps
        face = _FACE_FLOPS[d] * d * cells
        if kind == "adjoint":  # forward once, then the products of its transpose (about twice a forward)
            bytes_ += 2 * state * stages * 3
            flops += 3 * face * stages
        else:
            bytes_ += 2 * state * stages
            flops += face * stages
        if kind in ("batch", "hostrun", "adjoint", "hstep"):
            bytes_ += 2 * state
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------- plain restatement, 64 bits
def _prim(U):
    r, v = U[0], U[1:-1] / U[0]
    return torch.cat([r[None], v, ((G - 1) * r * (U[-1] / r - 0.5 * (v * v).sum(0)))[None]])


def _interp(scheme, a, b, c, d, e):
    """The value between c and d from five upwind-ordered values."""
    sm = lambda s, t: s * s + 0.25 * t * t  # noqa: E731
    b0 = sm(a - 2 * b + c, a - 4 * b + 3 * c)
    b1 = sm(b - 2 * c + d, b - d)
    b2 = sm(c - 2 * d + e, 3 * c - 4 * d + e)
    if scheme in ("wcns5", "wenoz"):
        if scheme == "wcns5":
            w = [k / (1e-6 + s) ** 2 for k, s in zip((1 / 16, 5 / 8, 5 / 16), (b0, b1, b2))]
        else:
            tau = (b2 - b0).abs()
            w = [k * (1 + (tau / (s + 1e-40)) ** 2) for k, s in zip((1 / 16, 5 / 8, 5 / 16), (b0, b1, b2))]
        u = ((3 * a - 10 * b + 15 * c) / 8, (-b + 6 * c + 3 * d) / 8, (3 * c + 6 * d - e) / 8)
        return sum(p * q for p, q in zip(w, u)) / (w[0] + w[1] + w[2])
    tau = (b2 - b0).abs()
    with torch.no_grad():  # the cut-off decisions are frozen
        if scheme == "teno":
            m = [(1 + tau / (s + 1e-40)) ** 6 for s in (b0, b1, b2)]
            cut = [k < 1e-5 * (m[0] + m[1] + m[2]) for k in m]
        else:
            ct, low = 0.15704178024750198, torch.minimum(b0, torch.minimum(b1, b2))
            cut = [tau * low < (ct * tau - (1 - ct) * low) * s for s in (b0, b1, b2)]
        flag = cut[0].long() + 2 * cut[1].long() + 4 * cut[2].long()
    T = [[3 / 128, -5 / 32, 45 / 64, 15 / 32, -5 / 128], [0, -1 / 16, 9 / 16, 9 / 16, -1 / 16],
         [0, 0, 3 / 8, 3 / 4, -1 / 8], [0, 0, 3 / 8, 3 / 4, -1 / 8], [1 / 16, -5 / 16, 15 / 16, 5 / 16, 0],
         [0, -1 / 8, 3 / 4, 3 / 8, 0], [3 / 8, -5 / 4, 15 / 8, 0, 0], [0, 0, 1, 0, 0]]
    w = torch.tensor(T, dtype=a.dtype, device=a.device).t()
    return sum(w[k][flag] * q for k, q in enumerate((a, b, c, d, e)))


def _faces(scheme, V, ax):
    """Left and right face states (prim) from prim with four ghosts along the last dim."""
    nv = V.shape[0]
    D = nv - 2
    U = _cons(V)
    m = V.shape[-1] - 5
    st = [U[..., k:k + m] for k in range(6)]
    L, R = V[..., 2:2 + m], V[..., 3:3 + m]
    H = lambda P: 0.5 * (P[1:-1] ** 2).sum(0) + P[-1] / P[0] * G / (G - 1)  # noqa: E731
    wl, wr = L[0].sqrt(), R[0].sqrt()
    vel = (wl * L[1:-1] + wr * R[1:-1]) / (wl + wr)
    ht = (wl * H(L) + wr * H(R)) / (wl + wr)
    ek = 0.5 * (vel * vel).sum(0)
    h = ht - ek
    c = ((G - 1) * h).sqrt()
    vn, tang = vel[ax], [i for i in range(D) if i != ax]
    scale = h if D == 1 else torch.ones_like(h)
    ends = [torch.zeros_like(L), torch.zeros_like(L)]

    def field(q, right):
        for side, args in ((0, q[0:5]), (1, q[5:0:-1])):
            z = _interp(scheme, *args)
            ends[side] = ends[side] + torch.stack([z * r if torch.is_tensor(r) or r else torch.zeros_like(z) for r in right])

    for s in (-1.0, 1.0):  # acoustic waves
        row = [(ek / h - s * vn / c) / 2] + [((s / c if i == ax else 0.0) - vel[i] / h) / 2 for i in range(D)] + [0.5 / h]
        field([sum(w * x for w, x in zip(row, S)) for S in st],
              [1.0] + [vel[i] + (s * c if i == ax else 0.0) for i in range(D)] + [h + ek + s * vn * c])
    field([((h - ek) * S[0] + sum(vel[i] * S[1 + i] for i in range(D)) - S[-1]) / scale for S in st],
          [scale / h] + [vel[i] * scale / h for i in range(D)] + [ek * scale / h])
    for i in tang:  # shear waves
        field([S[1 + i] - vel[i] * S[0] for S in st],
              [0.0] + [1.0 if k == i else 0.0 for k in range(D)] + [vel[i]])
    out = []
    for W in ends:
        v = W[1:-1] / W[0]
        out.append(torch.cat([W[0][None], v, ((G - 1) * (W[-1] - 0.5 * W[0] * (v * v).sum(0)))[None]]))
    fl, fr = out
    if D > 1:  # the solver's fallback, with its mix of right density and left velocity
        bad = (fl[0] < 0) | (fl[-1] < 0)
        fl = torch.where(bad, L, fl)
        bad = (fr[0] < 0) | (fr[-1] < 0)
        fr = torch.where(bad, torch.cat([R[:1], L[1:-1], R[-1:]]), fr)
    return fl, fr


def _flux(P, ax):
    vn = P[1 + ax]
    F = torch.stack([P[0] * vn] + [P[0] * P[1 + i] * vn + (P[-1] if i == ax else 0.0) for i in range(P.shape[0] - 2)] +
                    [(0.5 * P[0] * (P[1:-1] ** 2).sum(0) + G / (G - 1) * P[-1]) * vn])
    return F


def _hllc(L, R, ax):
    (rl, pl, ul), (rr, pr, ur) = ((P[0], P[-1], P[1 + ax]) for P in (L, R))
    cl, cr = (G * pl / rl).sqrt(), (G * pr / rr).sqrt()
    if L.shape[0] == 3:
        SL, SR = torch.minimum(ul - cl, ur - cr), torch.maximum(ul + cl, ur + cr)
    else:
        ps = ((pl + pr) / 2 - (rl + rr) / 2 * (cl + cr) / 2 * (ur - ul) / 2).clamp(min=0.0)
        q = lambda p: torch.where(ps <= p, torch.ones_like(p), (1 + (G + 1) / (2 * G) * (ps / p - 1)).clamp(min=1.0).sqrt())  # noqa: E731
        SL, SR = ul - cl * q(pl), ur + cr * q(pr)
    S = (pr - pl + rl * ul * (SL - ul) - rr * ur * (SR - ur)) / (rl * (SL - ul) - rr * (SR - ur))

    def star(P, SK):
        r, p, u = P[0], P[-1], P[1 + ax]
        U = _cons(P)
        f = r * (SK - u) / (SK - S)
        E = U[-1] / r + (S - u) * (S + p / (r * (SK - u)))
        W = torch.stack([f] + [f * (S if i == ax else P[1 + i]) for i in range(P.shape[0] - 2)] + [f * E])
        return _flux(P, ax) + SK * (W - U)

    FL, FR = star(L, SL), star(R, SR)
    F = torch.where(S > 0, FL, torch.where(S == 0, 0.5 * (FL + FR), FR))
    return torch.where(SL > 0, _flux(L, ax), torch.where((S > 0) | (S == 0) | (SR > 0), F, _flux(R, ax)))


def _roe(L, R, ax):
    D = L.shape[0] - 2
    H = lambda P: 0.5 * (P[1:-1] ** 2).sum(0) + P[-1] / P[0] * G / (G - 1)  # noqa: E731
    wl, wr = L[0].sqrt(), R[0].sqrt()
    v = (wl * L[1:-1] + wr * R[1:-1]) / (wl + wr)
    h = (wl * H(L) + wr * H(R)) / (wl + wr)
    q2 = 0.5 * (v * v).sum(0)
    c2 = (G - 1) * (h - q2)
    c, rho, vn = c2.sqrt(), wl * wr, v[ax]
    eps = (0.1 if D == 1 else 0.05) * (vn.abs() + c)
    lam = [torch.where(x.abs() < eps, (x * x + eps * eps) / (2 * eps), x.abs()) for x in (vn - c, vn, vn + c)]
    dr, dp, dv = R[0] - L[0], R[-1] - L[-1], R[1:-1] - L[1:-1]
    a = [lam[0] * (dp - rho * c * dv[ax]) / (2 * c2), lam[1] * (dr - dp / c2), lam[2] * (dp + rho * c * dv[ax]) / (2 * c2)]
    shear = [lam[1] * rho * (dv[i] if i != ax else torch.zeros_like(vn)) for i in range(D)]
    d = [a[0] + a[1] + a[2]]
    d += [a[0] * (v[i] - (c if i == ax else 0.0)) + a[2] * (v[i] + (c if i == ax else 0.0)) + a[1] * v[i] + shear[i]
          for i in range(D)]
    d += [a[0] * (h - c * vn) + a[2] * (h + c * vn) + a[1] * q2 + sum(v[i] * shear[i] for i in range(D))]
    return 0.5 * (_flux(L, ax) + _flux(R, ax) - torch.stack(d))


def _ghosts(case, V, ax, h, t):
    """Four ghosts on each side along the last dim (the sweep axis)."""
    if case["bc"] == "wrap":
        return torch.cat([V[..., -4:], V, V[..., :4]], -1)
    lo, hi = V[..., :1].expand(*V.shape[:-1], 4), V[..., -1:].expand(*V.shape[:-1], 4)
    if case["bc"] == "dmr":
        post = torch.tensor(_dmr_post(), device=V.device, dtype=V.dtype)
        if ax == 0:
            lo = post[:, None, None].expand_as(lo)
        else:
            x = (torch.arange(V.shape[1], device=V.device, dtype=V.dtype) + 0.5) * h
            mirror = V[..., :4].flip(-1) * torch.tensor([1.0, 1.0, -1.0, 1.0], device=V.device)[:, None, None]
            lo = torch.where((x < 1.0 / 6.0)[None, :, None], post[:, None, None], mirror)
            y = -h / 2 + torch.arange(4, device=V.device, dtype=V.dtype) * h
            behind = y[None, :] > math.sqrt(3.0) * (x[:, None] - (1 / 6 + math.sqrt(3.0) / 3 * (1 + 20 * t)))
            pre = torch.tensor([1.4, 0.0, 0.0, 1.0], device=V.device, dtype=V.dtype)
            hi = torch.where(behind[None], post[:, None, None], pre[:, None, None])
    return torch.cat([lo, V, hi], -1)


def _rhs(case, U, h, t=0.0):
    V = _prim(U)
    D = U.shape[0] - 2
    out = torch.zeros_like(U)
    for ax in range(D):
        W = _ghosts(case, V.movedim(-1 - ax, -1), ax, h, t)
        n = W.shape[-1] - 8
        L, R = _faces(case["scheme"], W, ax)
        F = (_hllc if case["flux"] == "hllc" else _roe)(L, R, ax)
        N = _flux(W, ax)
        d = (-0.3 * (N[..., 5:5 + n] - N[..., 3:3 + n]) + 1.5 * (F[..., 2:2 + n] - F[..., 1:1 + n]) +
             (F[..., 3:3 + n] - F[..., :n]) / 30) / h
        out = out + d.movedim(-1, -1 - ax)
    return out


def _rk3(case, U, h, dt, t=0.0):
    """One SSP-RK3 step and the last stage's right-hand side."""
    U1 = U - dt * _rhs(case, U, h, t)
    U2 = 0.75 * U + 0.25 * (U1 - dt * _rhs(case, U1, h, t + dt))
    r = _rhs(case, U2, h, t + dt / 2)
    return U / 3 + 2 / 3 * (U2 - dt * r), r


def _cfl_dt(case, U, h):
    V = _prim(U)
    c = (G * V[-1] / V[0]).sqrt()
    return case["cfl"] / sum(float((c + V[1 + d].abs()).max()) / h for d in range(V.shape[0] - 2))


def _steps(case, U, h):
    t, dts, linf = 0.0, [], []
    for _ in range(case["steps"]):
        dt = _cfl_dt(case, U, h)
        U, r = _rk3(case, U, h, dt, t)
        t += dt
        dts.append(dt)
        linf.append(float(r[0].abs().max()))
    return U, t, np.array(dts), np.array(linf)


def _host(U):
    return torch.from_numpy(_aos(U))


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        got = []
        for i, m in enumerate(_sizes(case, seed)):
            got.append(_steps(case, _initial(case, (m, m), seed * 1000 + i), 1.0 / m))
        return {"t": np.array([g[1] for g in got]), "steps": None, "cons": [_host(g[0]) for g in got]}
    n = _cells(case)
    h = _extent(case) / n[0]
    U = _initial(case, n, seed)
    if kind == "rhs":
        return _rhs(case, U, h)
    if kind == "adjoint":
        dt = float(_adjoint_dt(case, n))
        g = torch.from_numpy(_gen(seed + 77).normal(size=(math.prod(n), 4))).to(DEV).t().reshape(U.shape)
        states = [U]
        for _ in range(case["steps"]):
            with torch.no_grad():
                states.append(_rk3(case, states[-1], h, dt)[0])
        for W in reversed(states[:-1]):
            W = W.detach().requires_grad_(True)
            g, = torch.autograd.grad(_rk3(case, W, h, dt)[0], W, grad_outputs=g)
        return {"gradient": _host(g), "cons": _host(states[-1])}
    U, t, dts, linf = _steps(case, U, h)
    if kind == "run":
        return {"dt": dts, "linf": linf, "state": U}
    if kind == "hostrun":
        return {"dt": dts, "linf": linf, "cons": _host(U), "t": t}
    return {"cons": _host(U), "t": t, "dt": float(dts[0])}
