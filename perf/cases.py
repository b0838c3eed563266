"""Workloads of the finite-difference library: the calls a simulation program makes, with
their inputs, over the sizes that the library is used at.

``listed()`` names the standing cases, ``draw(rng)`` gives further ones of the same ranges,
``prepare`` makes a case's inputs and modules from a seed, ``run`` is one pass through the
public entry points, ``work`` counts the bytes and operations a pass cannot do without, and
``exact`` is the same computation in float64 with plain torch.

Sizes are interior extents; every field carries its ghost layers (order/2 of them).
"""
import math

import torch
import torch.nn.functional as F

import pde_module_b200 as P

F64 = torch.float64


# ---- the cases ------------------------------------------------------------------------
def listed():
    return [
        # The module loop of a 2D heat script (boundary, Laplacian, Euler), one step: the
        # smallest calls the library gets, where launches and host work count.
        dict(name="chain_256", kind="chain", nx=256, ny=256, order=2, bc="dirichlet"),
        # The same equation advanced by the fused rollout: the 256^2 heat workload.
        dict(name="heat2d_256", kind="heat2d", nx=256, ny=256, order=2, bc="dirichlet", steps=1000),
        # A plate of odd sides with insulated and held edges, fourth order.
        dict(name="heat2d_515x331_o4", kind="heat2d", nx=515, ny=331, order=4, bc="mixed", steps=300),
        # One operator on a large 3D scalar field (the 512^3 operator sweep).
        dict(name="lap3d_512", kind="operator", op="laplacian", nx=512, ny=512, nz=512, order=2),
        # A gradient on a ragged 3D box, fourth order: sides that no tile divides.
        dict(name="grad3d_ragged_o4", kind="operator", op="grad", nx=301, ny=255, nz=189, order=4),
        # A 3D heat rollout of a few steps between two outputs.
        dict(name="heat3d_256", kind="heat3d", nx=256, ny=192, nz=320, order=2, bc="dirichlet", steps=20),
        # The lid-driven cavity at its workload size: 50 Jacobi sweeps and a projection per step.
        dict(name="cavity_1024", kind="cavity", n=1024, steps=20),
        # The weakly compressible cavity of the reference's RK2 example (201 nodes a side).
        dict(name="wc_cavity_201", kind="wc", n=201, steps=100),
        # A parameter study: 64 uneven grids with their own diffusivities in one batch.
        dict(name="batch_heat_64", kind="batch_heat", grids=64, lo=64, hi=1024, steps=100),
        # The same for waves, fewer grids.
        dict(name="batch_wave_24", kind="batch_wave", grids=24, lo=64, hi=1024, steps=200),
        # Full-waveform inversion: one forward and one adjoint pass of the 512^2 wave workload.
        dict(name="wave_grad_512", kind="wave_grad", nx=512, ny=512, steps=2000),
        # Identifying a diffusivity field: forward and adjoint of a 256^2 heat rollout.
        dict(name="heat_grad_256", kind="heat_grad", nx=256, ny=256, order=2, bc="dirichlet", steps=1000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chain", "heat2d", "operator", "heat3d", "cavity", "wc", "batch_heat", "batch_wave", "wave_grad",
                       "heat_grad"])
    bc, order = rng.choice(["dirichlet", "mixed"]), rng.choice([2, 4])
    if kind == "chain":
        return dict(kind=kind, nx=_log(rng, 32, 1024), ny=_log(rng, 32, 1024), order=order, bc=bc)
    if kind == "heat2d":
        return dict(kind=kind, nx=_log(rng, 64, 1024), ny=_log(rng, 64, 1024), order=order, bc=bc,
                    steps=_log(rng, 100, 1000))
    if kind == "operator":
        return dict(kind=kind, op=rng.choice(["laplacian", "grad", "divergence"]), nx=_log(rng, 48, 512),
                    ny=_log(rng, 48, 512), nz=_log(rng, 48, 512), order=order)
    if kind == "heat3d":
        return dict(kind=kind, nx=_log(rng, 48, 320), ny=_log(rng, 48, 320), nz=_log(rng, 48, 320), order=order, bc=bc,
                    steps=rng.randint(4, 20))
    if kind == "cavity":
        return dict(kind=kind, n=_log(rng, 96, 1024), steps=rng.randint(5, 20))
    if kind == "wc":
        return dict(kind=kind, n=_log(rng, 65, 1025), steps=_log(rng, 20, 100))
    if kind == "batch_heat":
        return dict(kind=kind, grids=_log(rng, 8, 64), lo=64, hi=_log(rng, 256, 1024), steps=rng.randint(50, 100))
    if kind == "batch_wave":
        return dict(kind=kind, grids=_log(rng, 8, 24), lo=64, hi=_log(rng, 256, 1024), steps=rng.randint(50, 200))
    if kind == "wave_grad":
        return dict(kind=kind, nx=_log(rng, 96, 512), ny=_log(rng, 96, 512), steps=_log(rng, 200, 2000))
    return dict(kind=kind, nx=_log(rng, 64, 320), ny=_log(rng, 64, 320), order=order, bc=bc, steps=_log(rng, 200, 1000))


# ---- inputs (no code of the library) ------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _smooth(shape, gen, sigma):
    """Gaussian-filtered standard normal noise of a 2D shape, largest magnitude 1."""
    f = torch.randn(shape, device="cuda", generator=gen)
    kx = torch.fft.fftfreq(shape[0], device="cuda")[:, None]
    ky = torch.fft.rfftfreq(shape[1], device="cuda")[None, :]
    f = torch.fft.irfft2(torch.fft.rfft2(f) * torch.exp(-2.0 * (math.pi * sigma) ** 2 * (kx * kx + ky * ky)), s=shape)
    return (f / f.abs().max()).contiguous()


def _wrap_ghosts(f, g):
    """Periodic ghosts of the three leading axes."""
    for a in range(3):
        n = f.shape[a]
        idx = (torch.arange(n, device=f.device) - g) % (n - 2 * g) + g
        f = f.index_select(a, idx)
    return f.contiguous()


def _groups(bc):
    """(faces, is_dirichlet, value) of the heat cases."""
    if bc == "dirichlet":
        return [("ALL", True, 0.0)]
    return [("ALL", False, 0.0), ("-X", True, 0.25), ("+Y", True, 1.0)]


def _boundary(field, dx, g, bc):
    b = P.GridBoundary(field, dx, g)
    for faces, dirichlet, value in _groups(bc):
        (b.dirichlet_BC if dirichlet else b.vonNeumann_BC)(faces, value)
    return b


def _batch_sides(case, seed):
    import random
    r = random.Random(int(seed))
    return [(r.randint(case["lo"], case["hi"]), r.randint(case["lo"], case["hi"])) for _ in range(case["grids"])]


def _batch_sizes_of_case(case):
    """Grid sides belong to the case, not to the seed: a study keeps its grids and changes its fields."""
    return _batch_sides(case, 1000 * case["grids"] + case["hi"])


def _wc_cfl(n):
    """0.8 as in the reference's example at 201 nodes; finer grids at Re = 100 are bound by viscosity
    (nu dt / dx^2 stays at its value of 201 nodes), coarser ones by sound."""
    return 0.8 * min(1.0, 201.0 / n)


def _f32(x):
    return float(torch.tensor(x, dtype=torch.float32))


def _inputs(case, seed):
    gen, kind = _gen(seed), case["kind"]
    rand = lambda *s: torch.rand(s, device="cuda", generator=gen)  # noqa: E731
    if kind in ("chain", "heat2d", "heat3d", "heat_grad"):
        g = case["order"] // 2
        n = [case["nx"], case["ny"]] + ([case["nz"]] if kind == "heat3d" else [])
        shape = [s + 2 * g for s in n] + ([] if kind == "heat3d" else [1])
        dx = 1.0 / n[0]
        d = dict(g=g, dx=dx, dt=_f32((0.15 if len(n) == 2 else 0.1) * dx * dx), u=rand(*shape, 1))
        if kind == "heat_grad":
            d["alpha"] = (0.75 + 0.25 * _smooth(shape[:2], gen, 8.0))[:, :, None, None].contiguous()
            d["target"] = rand(*shape, 1)
        return d
    if kind == "operator":
        g = case["order"] // 2
        c = 3 if case["op"] == "divergence" else 1
        u = torch.randn([case[k] + 2 * g for k in ("nx", "ny", "nz")] + [c], device="cuda", generator=gen)
        return dict(g=g, dx=1.0 / case["nx"], u=_wrap_ghosts(u, g))
    if kind in ("cavity", "wc"):
        n = case["n"] + 2
        s = _smooth((n, n), gen, n / 16.0)  # stream function of the initial flow
        u = torch.stack([torch.roll(s, -1, 1) - torch.roll(s, 1, 1), torch.roll(s, 1, 0) - torch.roll(s, -1, 0)], -1)
        u = 0.3 * u / u.abs().max()
        d = dict(u=u[:, :, None, :].contiguous())
        if kind == "wc":
            d["rho"] = (1.0 + 0.01 * _smooth((n, n), gen, n / 16.0))[:, :, None, None].contiguous()
        return d
    if kind in ("batch_heat", "batch_wave"):
        sides = _batch_sizes_of_case(case)
        par = torch.rand(len(sides), generator=torch.Generator().manual_seed(int(seed))).tolist()
        if kind == "batch_heat":
            alpha = [_f32(math.exp(math.log(1e-3) * p)) for p in par]
            dx = [1.0 / x for x, _ in sides]
            return dict(dx=dx, alpha=alpha, dt=[_f32(0.2 * h * h / a) for h, a in zip(dx, alpha)],
                        u=[rand(x + 2, y + 2, 1, 1) for x, y in sides])
        K = [_f32((0.3 + 0.3 * p) ** 2 / (x - 1) ** 2) for p, (x, _) in zip(par, sides)]
        u, v = [], []
        for x, y in sides:
            f = torch.zeros(x + 2, y + 2, 1, 1, device="cuda")
            f[2:-2, 2:-2, 0, 0] = _smooth((x - 2, y - 2), gen, 6.0)
            u.append(f)
            v.append(f.clone())
        return dict(dx=[1.0 / (x - 1) for x, _ in sides], K=K, u=u, prev=v)
    # wave_grad: nodes on the unit square's long side, Ricker source at the centre, CFL 0.5
    shape = (case["nx"] + 2, case["ny"] + 2)
    dx = 1.0 / (case["nx"] - 1)
    c = 1.0 + 0.1 * _smooth(shape, gen, 8.0)
    dt = 0.5 * dx / (math.sqrt(2.0) * 1.1)
    t = torch.arange(case["steps"], dtype=F64) * dt
    a = (math.pi * (t - 1.2 * 10.0 * dx) / (10.0 * dx)) ** 2
    src = ((dt * dt / (dx * dx)) * (1.0 - 2.0 * a) * torch.exp(-a)).float().cuda()
    mask = torch.zeros(shape + (1, 1), device="cuda")
    mask[2:-2, 2:-2] = 1.0
    u0 = 0.1 * _smooth(shape, gen, 8.0)[:, :, None, None] * mask
    return dict(dx=dx, dt=dt, c=c[:, :, None, None].contiguous(), src=src, cell=(shape[0] // 2, shape[1] // 2),
                u0=u0.contiguous(), mask=mask, target=(0.1 * _smooth(shape, gen, 8.0)[:, :, None, None] * mask).contiguous())


# ---- what a program has in hand before the call ----------------------------------------------
def prepare(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    s = dict(kind=kind, case=case, d=d)
    if kind == "chain":
        s["bc"] = _boundary(d["u"], d["dx"], d["g"], case["bc"])
        s["lap"], s["euler"] = P.Laplacian(1, d["dx"], d["g"], order=case["order"]), P.ForwardEuler()
    elif kind in ("heat2d", "heat3d"):
        s["roll"] = P.HeatRollout(_boundary(d["u"], d["dx"], d["g"], case["bc"]), d["dx"], 1.0, d["dt"], case["order"])
    elif kind == "operator":
        shape, dx, g, o = tuple(d["u"].shape), d["dx"], d["g"], case["order"]
        s["op"] = {"laplacian": lambda: P.Laplacian(1, dx, g, order=o), "grad": lambda: P.Grad(1, shape, dx, g, order=o),
                   "divergence": lambda: P.Divergence(3, shape, dx, g, order=o)}[case["op"]]()
    elif kind == "cavity":
        s["solver"] = P.FractionalStepLDC(n=case["n"], Re=100.0, jacobi_iters=50)
        s["solver"].u.copy_(d["u"])
    elif kind == "wc":
        s["solver"], _, _ = P.lid_driven_cavity_wc(case["n"], cfl=_wc_cfl(case["n"]))
        s["m"] = (d["rho"] * d["u"]).contiguous()
    elif kind == "batch_heat":
        s["roll"] = P.BatchedHeatRollout(d["u"], d["dx"], d["alpha"], d["dt"])
    elif kind == "batch_wave":
        s["roll"] = P.BatchedWaveRollout(d["u"], d["prev"], d["dx"], d["K"])
    elif kind == "wave_grad":
        s["solver"] = P.WaveSolver(d["c"].shape[:2] + (1,), d["dx"], case["steps"], src=d["src"], src_cell=d["cell"])
    else:
        s["solver"] = P.HeatSolver(_boundary(d["u"], d["dx"], d["g"], case["bc"]), d["dx"], d["dt"], case["steps"],
                                   case["order"])
    return s


def run(s):
    kind, case, d = s["kind"], s["case"], s["d"]
    if kind == "chain":
        u2 = s["bc"](d["u"])
        return s["euler"](u2, s["lap"](u2, 1.0), d["dt"])
    if kind in ("heat2d", "heat3d"):
        return s["roll"](d["u"], case["steps"])
    if kind == "operator":
        return s["op"](d["u"], 0.7)
    if kind == "cavity":
        return s["solver"].step(case["steps"])
    if kind == "wc":
        return s["solver"](s["m"], d["rho"], case["steps"])
    if kind == "batch_heat":
        return s["roll"](case["steps"])
    if kind == "batch_wave":
        s["roll"](case["steps"])
        return s["roll"].fields + s["roll"].prev
    if kind == "wave_grad":
        c, u0 = d["c"].requires_grad_(True), d["u0"].requires_grad_(True)
        u = P.wave_rollout((d["dt"] * d["dt"]) * c * c, u0, s["solver"])
        loss = (((u - d["target"]) * d["mask"]) ** 2).mean()
        return (u.detach(),) + torch.autograd.grad(loss, (c, u0))
    alpha, u0 = d["alpha"].requires_grad_(True), d["u"].requires_grad_(True)
    u = P.heat_rollout(alpha, u0, s["solver"])
    loss = ((u - d["target"]) ** 2).mean()
    return (u.detach(),) + torch.autograd.grad(loss, (alpha, u0))


# ---- what a pass cannot do without ------------------------------------------------------------
def work(case):
    """Bytes: every input read once, every output written once.  Operations: those of the update
    formulas with like terms shared (order 2 in 2D: 9 per cell of a heat step), per cell and step."""
    kind = case["kind"]
    if kind in ("chain", "heat2d", "heat_grad", "heat3d"):
        dims = 3 if kind == "heat3d" else 2
        cells = case["nx"] * case["ny"] * (case["nz"] if dims == 3 else 1)
        lap = (2 * dims + 2) if case["order"] == 2 else (4 * dims + 3)  # shared products, sums
        per = lap + 3
        steps = case.get("steps", 1)
        if kind == "heat_grad":  # forward, and the adjoint with its gradient term
            return dict(bytes=4 * cells * 6, flops=cells * steps * (per + per + 2))
        return dict(bytes=8 * cells, flops=cells * steps * per)
    if kind == "operator":
        cells = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=(8 if case["op"] == "laplacian" else 16) * cells,
                    flops=cells * (9 if case["order"] == 2 else 15))
    if kind == "cavity":
        cells = case["n"] ** 2
        return dict(bytes=2 * 12 * cells, flops=cells * case["steps"] * (50 * 5 + 50))
    if kind == "wc":
        cells = case["n"] ** 2
        return dict(bytes=2 * 12 * cells, flops=cells * case["steps"] * 2 * 70)
    if kind in ("batch_heat", "batch_wave"):
        cells = sum(x * y for x, y in _batch_sizes_of_case(case))
        heat = kind == "batch_heat"
        return dict(bytes=(8 if heat else 16) * cells, flops=cells * case["steps"] * 9)
    cells = case["nx"] * case["ny"]
    return dict(bytes=4 * cells * 6, flops=cells * case["steps"] * (9 + 13))


# ---- the same in float64, plain torch -----------------------------------------------------------
class _Fill:
    """The boundary fill as one affine gather: out = mul * u[src] + add (per cell and component)."""

    def __init__(self, shape, comps, groups, dx, g):
        dev = "cuda"
        n, nd = shape, len(shape)
        cells = torch.arange(math.prod(shape) * comps, device=dev).reshape(*shape, comps)
        src, mul, add = cells.clone(), torch.ones_like(cells, dtype=F64), torch.zeros_like(cells, dtype=F64)
        for faces, dirichlet, value, ids in groups:
            nodes = torch.zeros(shape, dtype=torch.bool, device=dev)
            for a in range(nd):
                for sign, at in (("-", g), ("+", n[a] - 1 - g)):
                    if faces in ("ALL", sign + "XYZ"[a]):
                        sl = [slice(g, m - g) for m in n]
                        sl[a] = at
                        nodes[tuple(sl)] = True
            if dirichlet:  # the node's input vector with the group's components replaced
                src[nodes], mul[nodes], add[nodes] = cells[nodes], 1.0, 0.0
            for c in ids:
                if dirichlet:
                    mul[..., c][nodes], add[..., c][nodes] = 0.0, value
                for a in range(nd):
                    for inc, at in ((1, g), (-1, n[a] - 1 - g)):
                        m = nodes.select(a, at)
                        src[..., c].select(a, at - inc)[m] = cells[..., c].select(a, at + inc)[m]
                        mul[..., c].select(a, at - inc)[m] = -1.0 if dirichlet else 1.0
                        add[..., c].select(a, at - inc)[m] = 2.0 * value if dirichlet else -2.0 * inc * dx * value
        self.src, self.mul, self.add = src.reshape(-1), mul, add

    def __call__(self, u):
        return self.mul * u.reshape(-1)[self.src].reshape(self.mul.shape) + self.add


def _shift(u, g, nd, axis, by):
    return u[tuple(slice(g + (by if a == axis else 0), u.shape[a] - g + (by if a == axis else 0)) for a in range(nd))]


_LAP = {2: ((-1, 1.0), (0, -2.0), (1, 1.0)), 4: ((-2, -1 / 12), (-1, 16 / 12), (0, -30 / 12), (1, 16 / 12), (2, -1 / 12))}
_D1 = {2: ((-1, -0.5), (1, 0.5)), 4: ((-2, 1 / 12), (-1, -8 / 12), (1, 8 / 12), (2, -1 / 12))}


def _lap(u, g, nd, dx, order=2):
    return sum(w * _shift(u, g, nd, a, t) for a in range(nd) for t, w in _LAP[order]) / (dx * dx)


def _d1(u, g, nd, axis, dx, order=2):
    return sum(w * _shift(u, g, nd, axis, t) for t, w in _D1[order]) / dx


def _pad(v, g, nd):
    return F.pad(v, (0,) * (2 * (v.dim() - nd)) + (g, g) * nd)


def _heat_steps(u, alpha, fill, g, nd, dx, dt, order, steps):
    a = alpha if not torch.is_tensor(alpha) else _shift(alpha, g, nd, 0, 0)
    for _ in range(steps):
        v = fill(u)
        u = v + _pad(dt * (a * _lap(v, g, nd, dx, order)), g, nd)
    return u


def exact(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    if kind in ("chain", "heat2d", "heat3d", "heat_grad"):
        nd, g, dx = (3 if kind == "heat3d" else 2), d["g"], d["dx"]
        u = d["u"].double() if nd == 3 else d["u"].double()[:, :, 0]
        fill = _Fill(u.shape[:nd], 1, [gr + ((0,),) for gr in _groups(case["bc"])], dx, g)
        if kind != "heat_grad":
            return _heat_steps(u, 1.0, fill, g, nd, dx, d["dt"], case["order"], case.get("steps", 1)).reshape(d["u"].shape)
        alpha = d["alpha"].double()[:, :, 0].requires_grad_(True)
        u.requires_grad_(True)
        out = _heat_steps(u, alpha, fill, g, nd, dx, d["dt"], case["order"], case["steps"])
        loss = ((out - d["target"].double()[:, :, 0]) ** 2).mean()
        return tuple(t.detach().reshape(d["u"].shape) for t in (out,) + torch.autograd.grad(loss, (alpha, u)))
    if kind == "operator":
        u, g, dx, o = d["u"].double(), d["g"], d["dx"], case["order"]
        if case["op"] == "laplacian":
            return _pad(0.7 * _lap(u, g, 3, dx, o), g, 3)
        if case["op"] == "grad":
            return _pad(torch.stack([0.7 * _d1(u, g, 3, a, dx, o) for a in range(3)], -1), g, 3)
        return _pad(0.7 * sum(_d1(u[..., a:a + 1], g, 3, a, dx, o) for a in range(3)), g, 3)
    if kind == "cavity":
        n, g = case["n"], 1
        dx, nu = 1.0 / (n - 1), 0.01
        dt = 0.2 * min(dx, dx * dx / (4.0 * nu))
        shape = (n + 2, n + 2)
        fu = _Fill(shape, 2, [("ALL", True, 0.0, (0, 1)), ("+Y", True, 1.0, (0,))], dx, g)
        fp = _Fill(shape, 1, [("ALL", False, 0.0, (0,))], dx, g)
        u, p = d["u"].double()[:, :, 0], torch.zeros(shape + (1,), dtype=F64, device="cuda")
        for _ in range(case["steps"]):
            u2 = fu(u)
            c = _shift(u2, g, 2, 0, 0)
            conv = _d1(u2, g, 2, 0, dx) * c[..., :1] + _d1(u2, g, 2, 1, dx) * c[..., 1:]
            us = fu(u2 + _pad(dt * (nu * _lap(u2, g, 2, dx) - conv), g, 2))
            rhs = (dx * dx / dt) * (_d1(us[..., :1], g, 2, 0, dx) + _d1(us[..., 1:], g, 2, 1, dx))
            for _ in range(50):
                p = fp(p)
                q = _shift(p, g, 2, 0, -1) + _shift(p, g, 2, 0, 1) + _shift(p, g, 2, 1, -1) + _shift(p, g, 2, 1, 1)
                p[g:-g, g:-g] = 0.25 * (q - rhs)
            pb = fp(p)
            u = us - _pad(dt * torch.cat([_d1(pb, g, 2, 0, dx), _d1(pb, g, 2, 1, dx)], -1), g, 2)
        return u[:, :, None], p[:, :, None]
    if kind == "wc":
        n, g = case["n"], 1
        dx, nu, cs = 1.0 / (n - 1), 0.01, 10.0
        cfl = _wc_cfl(n)
        dt = min(cfl * dx * dx / nu, cfl * dx / cs, cfl * dx / (cs + 1.0))
        eps = -0.01 * dx ** 4 / (dt * nu)
        shape = (n + 2, n + 2)
        fu = _Fill(shape, 2, [("ALL", True, 0.0, (0, 1)), ("+Y", True, 1.0, (0,))], dx, g)
        fr = _Fill(shape, 1, [("ALL", False, 0.0, (0,))], dx, g)

        def bc(m, r):
            u, r2 = fu(m / r), fr(r)
            return r2 * u, r2

        def f(m, r):
            u = m / r
            diff = _pad(nu * _lap(u, g, 2, dx), g, 2)
            conv = _d1(m * u[..., :1], g, 2, 0, dx) + _d1(m * u[..., 1:], g, 2, 1, dx)
            pr = cs * cs * (r - 1.0)
            dp = torch.cat([_d1(pr, g, 2, 0, dx), _d1(pr, g, 2, 1, dx)], -1)
            km = _pad(eps * _lap(diff, g, 2, dx) - dp - conv, g, 2) + diff
            return km, _pad(-(_d1(m[..., :1], g, 2, 0, dx) + _d1(m[..., 1:], g, 2, 1, dx)), g, 2)

        m, r = (d["rho"] * d["u"]).double()[:, :, 0], d["rho"].double()[:, :, 0]
        for _ in range(case["steps"]):
            m0, r0 = bc(m, r)
            km, kr = f(m0, r0)
            km, kr = f(*bc(m0 + dt / 2 * km, r0 + dt / 2 * kr))
            m, r = m0 + dt * km, r0 + dt * kr
        return m[:, :, None], r[:, :, None]
    if kind == "batch_heat":
        out = []
        for u, dx, a, dt in zip(d["u"], d["dx"], d["alpha"], d["dt"]):
            fill = _Fill(u.shape[:2], 1, [("ALL", True, 0.0, (0,))], dx, 1)
            out.append(_heat_steps(u.double()[:, :, 0], a, fill, 1, 2, dx, dt, 2, case["steps"])[:, :, None])
        return out
    if kind == "batch_wave":
        last, prev = [], []
        for u, v, dx, K in zip(d["u"], d["prev"], d["dx"], d["K"]):
            u, v = u.double()[:, :, 0], v.double()[:, :, 0]
            for _ in range(case["steps"]):
                u, v = 2.0 * u - v + _pad(K * _lap(u, 2, 2, dx), 2, 2), u
                u[:2], u[-2:], u[:, :2], u[:, -2:] = 0.0, 0.0, 0.0, 0.0
            last.append(u[:, :, None])
            prev.append(v[:, :, None])
        return last + prev
    c, u0 = d["c"].double()[:, :, 0].requires_grad_(True), d["u0"].double()[:, :, 0].requires_grad_(True)
    K = (d["dt"] * d["dt"]) * c * c
    Ki = _shift(K, 2, 2, 0, 0)
    point = torch.zeros(u0.shape, dtype=F64, device="cuda")
    point[d["cell"][0], d["cell"][1]] = 1.0
    point = point[2:-2, 2:-2]
    w, v = (u0 * d["mask"].double()[:, :, 0])[2:-2, 2:-2], None
    v = w
    for s in d["src"].double():
        full = _pad(w, 2, 2)
        w, v = 2.0 * w - v + Ki * _lap(full, 2, 2, d["dx"]) + s * point, w
    u = _pad(w, 2, 2)
    loss = (((u - d["target"].double()[:, :, 0]) * d["mask"].double()[:, :, 0]) ** 2).mean()
    return tuple(t.detach()[:, :, None] for t in (u,) + torch.autograd.grad(loss, (c, u0)))
