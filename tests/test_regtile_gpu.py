"""The register-tile 2D kernels against the float32 oracle, bit for bit, at the
sizes where their windows change shape: boxes of exactly one window, one strip or
one lane more or less, odd sides, one and several tiles per axis, both orders,
passes that end short, every kind of face group."""
import numpy as np
import pytest
import torch

from oracle import fdm
import pde_module_b200 as P

pytestmark = pytest.mark.gpu

DIRICHLET = [("ALL", 1, 0.5, (0,))]
MIXED = [("ALL", 2, 0.3, (0,)), ("-X", 1, 0.25, (0,)), ("+Y", 1, -1.0, (0,))]
NEUMANN = [("ALL", 2, -0.4, (0,))]

# interior sides (stencil box)
SIDES = [(8, 8), (9, 11), (16, 64), (17, 65), (63, 66), (64, 64), (65, 128), (96, 129), (130, 67), (201, 333)]


@pytest.mark.parametrize("sides", SIDES)
@pytest.mark.parametrize("order,spec", [(2, DIRICHLET), (2, MIXED), (2, NEUMANN), (4, DIRICHLET), (4, MIXED)])
def test_heat_rollout_window_edges(sides, order, spec):
    g = order // 2
    shape = (sides[0] + 2 * g, sides[1] + 2 * g, 1)
    dx = 1.0 / sides[0]
    dt = 0.15 * dx * dx
    u0 = np.random.default_rng(sides[0] * 1000 + sides[1] + order).random(shape + (1,)).astype(np.float32)
    ud = torch.from_numpy(u0).cuda()
    bc = P.GridBoundary(ud, dx, g)
    for name, typ, val, comps in spec:
        bc.set_BC(name, val, typ, comps)
    groups = fdm.standard_groups(shape, g, spec)
    for steps, k in ((1, 0), (11, 4), (27, 0)):
        got = P.HeatRollout(bc, dx, 0.9, dt, order=order, steps_per_pass=k)(ud, steps).cpu().numpy()
        ref = fdm.heat_rollout(u0, groups, dx, g, 0.9, dt, steps, order)
        assert np.array_equal(got, ref), (steps, k)
    assert np.array_equal(ud.cpu().numpy(), u0)


def test_heat_rollout_unfilled_ghosts_keep_the_shared_memory_path():
    """A face no group touches keeps its ghosts' input values."""
    shape, g = (40, 37, 1), 1
    dx = 1.0 / 38
    spec = [("-Y", 1, 0.4, (0,)), ("+X", 2, -0.3, (0,))]
    u0 = np.random.default_rng(5).random(shape + (1,)).astype(np.float32)
    ud = torch.from_numpy(u0).cuda()
    bc = P.GridBoundary(ud, dx, g)
    for name, typ, val, comps in spec:
        bc.set_BC(name, val, typ, comps)
    got = P.HeatRollout(bc, dx, 0.9, 0.15 * dx * dx)(ud, 13).cpu().numpy()
    assert np.array_equal(got, fdm.heat_rollout(u0, fdm.standard_groups(shape, g, spec), dx, g, 0.9, 0.15 * dx * dx, 13))


@pytest.mark.parametrize("n,iters,k", [(8, 5, 0), (17, 9, 3), (62, 50, 0), (64, 7, 7), (129, 50, 0), (300, 33, 8)])
def test_cavity_window_edges(n, iters, k):
    """Jacobi windows and the velocity kernels' tiles at one window, one lane or strip
    more, several tiles; passes of uneven depth; the residual of the last sweep."""
    s = P.FractionalStepLDC(n=n, Re=100.0, jacobi_iters=iters, jacobi_per_pass=k, dt=1e-3 / n)
    rng = np.random.default_rng(n)
    s.u.copy_(torch.from_numpy((0.1 * rng.standard_normal(tuple(s.u.shape))).astype(np.float32)))
    s.p.copy_(torch.from_numpy((0.1 * rng.standard_normal(tuple(s.p.shape))).astype(np.float32)))
    u, p = s.u.cpu().numpy(), s.p.cpu().numpy()
    s.step(2, residuals=True)
    G = fdm.exterior_groups(u.shape, 1)
    ug = [dict(ids=G["ALL"], type=1, value=0.0, comps=(0, 1)), dict(ids=G["+Y"], type=1, value=1.0, comps=(0,))]
    pg = [dict(ids=G["ALL"], type=2, value=0.0, comps=(0,))]
    for _ in range(2):
        u, p = fdm.ldc_step(u, p, ug, pg, s.dx, 1, s.nu, s.dt, iters)
    assert np.array_equal(s.u.cpu().numpy(), u)
    assert np.array_equal(s.p.cpu().numpy(), p)
    assert torch.isfinite(s.residuals[:2]).all() and (s.residuals[:2] > 0).all()


BOXES = [(16, 8), (64, 128), (65, 129), (63, 127), (72, 200), (130, 33), (97, 260)]


@pytest.mark.parametrize("k,nsteps", [(0, 23), (4, 9), (12, 1)])
@pytest.mark.parametrize("spec", [DIRICHLET, MIXED])
def test_batched_heat_window_edges(k, nsteps, spec):
    fields = [np.random.default_rng(7 + i).random((x + 2, y + 2, 1, 1)).astype(np.float32) for i, (x, y) in enumerate(BOXES)]
    dev = [torch.from_numpy(f).cuda() for f in fields]
    dx = [1.0 / x for x, _ in BOXES]
    alpha = [0.5 + 0.1 * i for i in range(len(BOXES))]
    dt = [float(np.float32(0.2 * h * h / a)) for h, a in zip(dx, alpha)]
    bc = P.GridBoundary(dev[0], dx[0], 1)
    for name, typ, val, comps in spec:
        bc.set_BC(name, val, typ, comps)
    boxes = BOXES[1:] if k == 12 else BOXES  # 16 rows do not hold a window with a halo of 12
    first = len(BOXES) - len(boxes)
    roll = P.BatchedHeatRollout(dev[first:], dx[first:], alpha[first:], dt[first:], boundary=bc, steps_per_pass=k)
    assert roll.plan.register_tiles == 1
    roll(nsteps)
    assert P._lib.device_error() == 0
    for i in range(first, len(BOXES)):
        ref = fdm.heat_rollout(fields[i], fdm.standard_groups(fields[i].shape[:3], 1, spec), dx[i], 1, alpha[i], dt[i], nsteps)
        assert np.array_equal(dev[i].cpu().numpy(), ref), BOXES[i]


@pytest.mark.parametrize("k,nsteps", [(0, 23), (4, 9), (8, 2)])
def test_batched_wave_window_edges(k, nsteps):
    boxes = [(x + 2, y + 2) for x, y in BOXES]  # the wave's box leaves out the node ring
    u = []
    for i, (x, y) in enumerate(boxes):
        f = np.zeros((x + 2, y + 2, 1, 1), dtype=np.float32)
        f[2:-2, 2:-2, 0, 0] = np.random.default_rng(70 + i).standard_normal((x - 2, y - 2))
        u.append(f)
    K = [float(np.float32(0.2 / (x * x))) for x, _ in boxes]
    dx = [1.0 / x for x, _ in boxes]
    now, prev = [torch.from_numpy(f).cuda() for f in u], [torch.from_numpy(f).cuda() for f in u]
    roll = P.BatchedWaveRollout(now, prev, dx, K, steps_per_pass=k)
    assert roll.plan.register_tiles == 1
    roll(nsteps)
    assert P._lib.device_error() == 0
    for i in range(len(boxes)):
        st = fdm.wave_forward(np.full(u[i].shape, K[i], np.float32), u[i], None, -1, nsteps, dx[i])
        assert np.array_equal(now[i].cpu().numpy()[:, :, 0, 0], st[-1]), boxes[i]
        assert np.array_equal(prev[i].cpu().numpy()[:, :, 0, 0], st[-2]), boxes[i]


@pytest.mark.parametrize("X,Y,g,N,k,every,src", [(12, 12, 1, 5, 0, None, None), (68, 132, 1, 21, 0, 7, (5, 60)),
                                                 (69, 133, 1, 21, 5, None, (30, 131)), (70, 203, 2, 17, 0, 6, (1, 1)),
                                                 (204, 67, 1, 30, 12, 12, (100, 33))])
def test_wave_window_edges(X, Y, g, N, k, every, src):
    """Forward and adjoint windows at even and odd sides (paired and single columns),
    one window, several, a source on an edge and on a ghost; against the oracle."""
    rng = np.random.default_rng(X + Y)
    dx = 1.0 / (X - 3)
    K = (0.1 * dx * dx * (1.0 + rng.random((X, Y, 1, 1)))).astype(np.float32)
    u0 = rng.standard_normal((X, Y, 1, 1)).astype(np.float32)
    grad = rng.standard_normal((X, Y, 1, 1)).astype(np.float32)
    s = (dx * dx * rng.random(N)).astype(np.float32)
    solver = P.WaveSolver((X, Y, 1), dx, N, src=torch.from_numpy(s).cuda() if src else None, src_cell=src, ghost_cells=g,
                          steps_per_pass=k, checkpoint_every=every)
    Kd = torch.from_numpy(K).cuda()
    uN = solver.forward(Kd, torch.from_numpy(u0).cuda())
    gK, gu = solver.backward(Kd, torch.from_numpy(grad).cuda())
    st = fdm.wave_forward(K, u0, s, src[0] * Y + src[1] if src else -1, N, dx, ghost=g)
    rgK, mu0, mu1 = fdm.wave_adjoint(K, st, grad, dx, ghost=g)
    assert np.array_equal(uN.cpu().numpy()[:, :, 0, 0], st[-1])
    assert np.array_equal(gK.cpu().numpy()[:, :, 0, 0], rgK)
    assert np.array_equal(gu.cpu().numpy()[:, :, 0, 0], mu0 - mu1)


@pytest.mark.parametrize("sides", [(8, 8), (9, 33), (64, 64), (65, 130), (203, 71)])
@pytest.mark.parametrize("spec", [DIRICHLET, MIXED, NEUMANN])
def test_heat_gradient_window_edges(sides, spec):
    """Forward with a diffusivity field and its adjoint: the transposed boundary fill at
    corners, one window and several, short passes; against the oracle."""
    X, Y = sides[0] + 2, sides[1] + 2
    rng = np.random.default_rng(X * Y)
    dx = 1.0 / sides[0]
    dt = 0.2 * dx * dx
    alpha = (0.5 + 0.5 * rng.random((X, Y, 1, 1))).astype(np.float32)
    u0 = rng.random((X, Y, 1, 1)).astype(np.float32)
    lam = rng.standard_normal((X, Y, 1, 1)).astype(np.float32)
    bc = P.GridBoundary(torch.from_numpy(u0).cuda(), dx, 1)
    for name, typ, val, comps in spec:
        bc.set_BC(name, val, typ, comps)
    groups = fdm.standard_groups((X, Y, 1), 1, spec)
    for N, k, every in ((1, 0, None), (14, 4, 6), (21, 0, None)):
        solver = P.HeatSolver(bc, dx, dt, N, steps_per_pass=k, checkpoint_every=every)
        a = torch.from_numpy(alpha).cuda()
        uN = solver.forward(a, torch.from_numpy(u0).cuda())
        ga, gu = solver.backward(a, torch.from_numpy(lam).cuda())
        ref, S = fdm.heat_forward_field(alpha, u0, groups, dx, 1, dt, N)
        rga, rgu = fdm.heat_adjoint(alpha, S, lam, groups, dx, 1, dt)
        assert np.array_equal(uN.cpu().numpy(), ref), N
        assert np.array_equal(ga.cpu().numpy(), rga), N
        assert np.array_equal(gu.cpu().numpy(), rgu), N


@pytest.mark.parametrize("shape,order", [((9, 8, 10), 2), ((5, 7, 6), 2), ((20, 33, 47), 2), ((34, 30, 132), 2),
                                         ((6, 137, 135), 2), ((20, 33, 47), 4), ((34, 30, 36), 4)])
@pytest.mark.parametrize("spec", [DIRICHLET, [("ALL", 2, 0.3, (0,)), ("-X", 1, 0.25, (0,)), ("+Z", 1, -1.0, (0,))],
                                  [("-Y", 1, 0.4, (0,)), ("+X", 2, -0.3, (0,))]])
def test_heat3d_streaming_fill(shape, order, spec):
    """The one-step 3D path on even and odd sides (its row maps), from three interior
    cells a side; the single-pass fill at faces, edges, corners and unfilled faces."""
    g = order // 2
    dx = 1.0 / shape[0]
    dt = 0.1 * dx * dx
    u0 = np.random.default_rng(sum(shape)).random(shape + (1,)).astype(np.float32)
    ud = torch.from_numpy(u0).cuda()
    bc = P.GridBoundary(ud, dx, g)
    for name, typ, val, comps in spec:
        bc.set_BC(name, val, typ, comps)
    groups = fdm.standard_groups(shape, g, spec)
    for steps in (1, 2, 5):
        got = P.HeatRollout(bc, dx, 0.9, dt, order=order)(ud, steps).cpu().numpy()
        assert np.array_equal(got, fdm.heat_rollout(u0, groups, dx, g, 0.9, dt, steps, order)), steps
    assert np.array_equal(ud.cpu().numpy(), u0)


@pytest.mark.parametrize("shape", [(7, 9), (95, 101), (203, 204), (242, 290), (331, 403), (520, 640)])
def test_weakly_compressible_tile_rule(shape):
    """The automatic tiles of the weakly compressible step at each of its sides (8, one
    per SM, 17, 24, 32) and their remainders, on a momentum that is only 4-byte aligned."""
    from oracle import acm
    from tests.test_wc_gpu import _case
    m, rho, md, rd, u_bc, r_bc, ug, rg, dx, nu, c2, rho0, eps, dt = _case(shape + (1,), 11)
    odd = torch.empty(md.numel() + 1, device="cuda")[1:].view(md.shape).copy_(md)
    got_m, got_r = P.WeaklyCompressibleRK2(u_bc, r_bc, dx, nu, c2, rho0, eps, dt)(odd, rd, 2)
    ref_m, ref_r = acm.wc_rk2(m, rho, ug, rg, dx, 1, nu, eps, c2, rho0, dt, 2)
    assert np.array_equal(got_m.cpu().numpy(), ref_m)
    assert np.array_equal(got_r.cpu().numpy(), ref_r)


# X*Y mod 4 = 1, 2, 3 and 0; rows of every length mod 4; tiles of one and of several
# row quadruples; z of one, two and three tiles
@pytest.mark.parametrize("shape", [(9, 9, 9), (7, 10, 11), (9, 11, 70), (11, 12, 67), (6, 35, 133), (10, 41, 187),
                                   (5, 130, 261)])
@pytest.mark.parametrize("order,extra", [(2, 0), (4, 0), (2, 1)])
def test_streaming_quad_rows(shape, order, extra):
    """The 3D operators on shapes whose rows arrive four apart, up to the array's last
    X*Y mod 4 rows."""
    g = order // 2 + extra
    rng = np.random.default_rng(shape[2] + order)
    u = rng.standard_normal(shape + (3,)).astype(np.float32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    s = u[..., :1]
    for n in (1, 3):
        got = P.Laplacian(n, 0.3, g, order=order)(dev(u[..., :n]), 0.7).cpu().numpy()
        assert np.array_equal(got, fdm.laplacian(u[..., :n], 0.3, g, 0.7, order)), n
    got = P.Grad(1, shape + (1,), 0.3, g, order=order)(dev(s), 0.7).cpu().numpy()
    assert np.array_equal(got, fdm.grad(s, 0.3, g, 0.7, order).reshape(got.shape))
    got = P.Divergence(3, shape + (3,), 0.3, g, order=order)(dev(u), 0.7).cpu().numpy()
    assert np.array_equal(got, fdm.divergence(u, 0.3, g, 0.7, order).reshape(got.shape))
