"""Batched rollouts (one persistent launch over a tile work queue) against the
per-grid fused rollout and the float32 oracle, bitwise, on uneven grids."""
import numpy as np
import pytest
import torch

from oracle import fdm
import pde_module_b200 as P

pytestmark = pytest.mark.gpu


def _grids(n, lo, hi, seed, g=1):
    rng = np.random.default_rng(seed)
    sides = rng.integers(lo, hi + 1, size=(n, 2))
    alpha = np.exp(rng.uniform(np.log(1e-3), 0.0, size=n))
    fields, dx, dts = [], [], []
    for i, (sx, sy) in enumerate(sides):
        shape = (int(sx) + 2 * g, int(sy) + 2 * g, 1, 1)
        fields.append(np.random.default_rng(100 + i).random(shape).astype(np.float32))
        h = 1.0 / (max(sx, sy) - 1)
        dx.append(h)
        dts.append(0.2 * h * h / alpha[i])
    return fields, dx, alpha.tolist(), dts


def _bc(u, dx, g, spec):
    bc = P.GridBoundary(u, dx, g)
    for name, typ, val, comps in spec:
        bc.set_BC(name, val, typ, comps)
    return bc


@pytest.mark.parametrize("tile,k,nsteps", [((32, 64), 8, 37), ((16, 32), 4, 9), ((64, 32), 6, 1),
                                           ((32, 32), 3, 2), ((24, 40), 5, 50)])
def test_batched_heat_matches_per_grid(tile, k, nsteps):
    g = 1
    fields, dx, alpha, dts = _grids(14, 5, 150, seed=7)
    spec = [("ALL", 1, 0.0, (0,))]
    dev = [torch.from_numpy(f).cuda() for f in fields]
    ref = []
    for i, u in enumerate(dev):
        bc = _bc(u, dx[i], g, spec)
        ref.append(P.HeatRollout(bc, dx[i], alpha[i], dts[i], steps_per_pass=k)(u, nsteps).cpu().numpy())
    batch = [u.clone() for u in dev]
    roll = P.BatchedHeatRollout(batch, dx, alpha, dts, tile=tile, steps_per_pass=k)
    roll(nsteps)
    torch.cuda.synchronize()
    assert P._lib.device_error() == 0
    for i in range(len(batch)):
        assert np.array_equal(batch[i].cpu().numpy(), ref[i]), f"grid {i} {fields[i].shape}"
    for i in (0, 3):
        o = fdm.heat_rollout(fields[i], fdm.standard_groups(fields[i].shape[:3], g, spec), dx[i], g, alpha[i],
                             dts[i], nsteps)
        assert np.array_equal(batch[i].cpu().numpy(), o)


def test_batched_heat_neumann_order4():
    g, order = 2, 4
    fields, dx, alpha, dts = _grids(9, 12, 90, seed=11, g=g)
    spec = [("ALL", 1, 0.0, (0,)), ("+X", 2, 0.75, (0,)), ("-Y", 2, -0.5, (0,))]
    dev = [torch.from_numpy(f).cuda() for f in fields]
    batch = [u.clone() for u in dev]
    bc0 = _bc(batch[0], dx[0], g, spec)
    roll = P.BatchedHeatRollout(batch, dx, alpha, dts, boundary=bc0, ghost_cells=g, order=order, tile=(32, 32),
                                steps_per_pass=4)
    roll(21)
    torch.cuda.synchronize()
    for i, u in enumerate(dev):
        bc = _bc(u, dx[i], g, spec)
        ref = P.HeatRollout(bc, dx[i], alpha[i], dts[i], order=order, steps_per_pass=4)(u, 21).cpu().numpy()
        assert np.array_equal(batch[i].cpu().numpy(), ref), f"grid {i}"
    o = fdm.heat_rollout(fields[2], fdm.standard_groups(fields[2].shape[:3], g, spec), dx[2], g, alpha[2], dts[2],
                         21, order)
    assert np.array_equal(batch[2].cpu().numpy(), o)


def test_batched_heat_graph_replay():
    fields, dx, alpha, dts = _grids(8, 30, 200, seed=5)
    a = [torch.from_numpy(f).cuda() for f in fields]
    b = [u.clone() for u in a]
    ra = P.BatchedHeatRollout(a, dx, alpha, dts, steps_per_pass=8)
    rb = P.BatchedHeatRollout(b, dx, alpha, dts, steps_per_pass=8)
    gr = ra.graph(20)
    gr.replay()
    gr.replay()
    rb(20)
    rb(20)
    torch.cuda.synchronize()
    for x, y in zip(a, b):
        assert torch.equal(x, y)


@pytest.mark.parametrize("tile,k,nsteps", [((32, 64), 8, 33), ((16, 16), 5, 12)])
def test_batched_wave_matches_oracle(tile, k, nsteps):
    rng = np.random.default_rng(21)
    n = 10
    sides = rng.integers(8, 120, size=(n, 2))
    fields, prev, dx, Ks, u0s = [], [], [], [], []
    for i, (sx, sy) in enumerate(sides):
        X, Y = int(sx) + 2, int(sy) + 2
        h = 1.0 / (max(X, Y) - 3)
        c = 1.0 + 0.5 * rng.random()
        dt = 0.5 * h / (np.sqrt(2.0) * c)
        K = np.float32(dt * dt * c * c)
        u0 = np.zeros((X, Y, 1, 1), dtype=np.float32)
        u0[2:-2, 2:-2, 0, 0] = rng.standard_normal((X - 4, Y - 4))
        u0s.append(u0)
        fields.append(torch.from_numpy(u0).cuda())
        prev.append(torch.from_numpy(u0).cuda())
        dx.append(h)
        Ks.append(float(K))
    roll = P.BatchedWaveRollout(fields, prev, dx, Ks, tile=tile, steps_per_pass=k)
    roll(nsteps)
    torch.cuda.synchronize()
    assert P._lib.device_error() == 0
    for i in range(n):
        Kf = np.full(u0s[i].shape, Ks[i], dtype=np.float32)
        st = fdm.wave_forward(Kf, u0s[i], None, None, nsteps, dx[i])
        assert np.array_equal(fields[i].cpu().numpy()[:, :, 0, 0], st[-1]), f"grid {i}"
        assert np.array_equal(prev[i].cpu().numpy()[:, :, 0, 0], st[-2]), f"grid {i}"


def test_batched_zero_steps_is_identity():
    fields, dx, alpha, dts = _grids(3, 10, 40, seed=1)
    a = [torch.from_numpy(f).cuda() for f in fields]
    P.BatchedHeatRollout(a, dx, alpha, dts)(0)
    for x, f in zip(a, fields):
        assert np.array_equal(x.cpu().numpy(), f)


@pytest.mark.parametrize("kind", ["heat", "wave"])
def test_batched_thin_grids_stay_in_their_work_buffer(kind):
    """Narrow boxes take more register tiles than shared-memory tiles: the words behind
    a work buffer of the size asked for stay as they are, and results match the oracle."""
    boxes = [(150, 50), (300, 61), (661, 25), (25, 25), (28, 57)] * 3
    pad = 1 if kind == "heat" else 2
    rng = np.random.default_rng(2)
    u = []
    for x, y in boxes:
        f = np.zeros((x + 2 * pad, y + 2 * pad, 1, 1), dtype=np.float32)
        f[pad:-pad, pad:-pad, 0, 0] = rng.random((x, y))
        u.append(f)
    dev, prev = [torch.from_numpy(f).cuda() for f in u], [torch.from_numpy(f).cuda() for f in u]
    dx = [1.0 / x for x, _ in boxes]
    dt = [float(np.float32(0.2 * h * h)) for h in dx]
    if kind == "heat":
        roll = P.BatchedHeatRollout(dev, dx, 1.0, dt)
    else:
        roll = P.BatchedWaveRollout(dev, prev, dx, dt)
    need = roll._work.numel()
    guarded = torch.full((need + 4096,), 0xA5, device="cuda", dtype=torch.uint8)
    roll._work = guarded[:need]
    roll.configure()
    assert roll.plan.register_tiles == 1 and 4 * roll.plan.total_tiles + 256 <= need
    roll(23)
    assert P._lib.device_error() == 0
    assert bool((guarded[need:] == 0xA5).all())
    for i in range(5):
        if kind == "heat":
            spec = fdm.standard_groups(u[i].shape[:3], 1, [("ALL", 1, 0.0, (0,))])
            assert np.array_equal(dev[i].cpu().numpy(), fdm.heat_rollout(u[i], spec, dx[i], 1, 1.0, dt[i], 23)), boxes[i]
        else:
            st = fdm.wave_forward(np.full(u[i].shape, dt[i], np.float32), u[i], None, None, 23, dx[i])
            assert np.array_equal(dev[i].cpu().numpy()[:, :, 0, 0], st[-1]), boxes[i]
            assert np.array_equal(prev[i].cpu().numpy()[:, :, 0, 0], st[-2]), boxes[i]


@pytest.mark.parametrize("rows,tile,k,register", [(24, None, 0, 0), (66, None, 0, 1), (24, None, 4, 1),
                                                  (24, (64, 64), 8, 0)])
@pytest.mark.parametrize("nsteps", [1, 2, 23])
@pytest.mark.parametrize("g", [1, 2])
def test_batched_wave_zeroes_the_ring(rows, tile, k, register, nsteps, g):
    """Fields that come in with values on the node ring and the ghosts: those count as 0
    and are 0 in both levels afterwards, on either kind of tile (22 rows of cells hold no
    window with a halo of 10)."""
    shapes = [(70, 90), (131, 40), (rows, 300)]
    rng = np.random.default_rng(g + nsteps)
    u = [rng.standard_normal((x + 2 * g, y + 2 * g, 1, 1)).astype(np.float32) for x, y in shapes]
    now, prev = [torch.from_numpy(f).cuda() for f in u], [torch.from_numpy(f).cuda() for f in u]
    dx = [1.0 / (x - 1) for x, _ in shapes]
    K = [float(np.float32(0.2 * h * h)) for h in dx]
    roll = P.BatchedWaveRollout(now, prev, dx, K, ghost_cells=g, tile=tile, steps_per_pass=k)
    assert roll.plan.register_tiles == register
    roll(nsteps)
    assert P._lib.device_error() == 0
    for i in range(len(shapes)):
        f = np.zeros_like(u[i])
        f[g + 1:-g - 1, g + 1:-g - 1] = u[i][g + 1:-g - 1, g + 1:-g - 1]
        st = fdm.wave_forward(np.full(f.shape, K[i], np.float32), f, None, None, nsteps, dx[i], ghost=g)
        assert np.array_equal(now[i].cpu().numpy()[:, :, 0, 0], st[-1]), shapes[i]
        assert np.array_equal(prev[i].cpu().numpy()[:, :, 0, 0], st[-2]), shapes[i]
