"""Fractional-step lid-driven cavity: fused kernels against the oracle's
composition of the operators (oracle/fdm.py: ldc_step), bitwise, on small grids
with several temporal-blocking depths of the Jacobi sweeps."""
import numpy as np
import pytest
import torch

from oracle import fdm
import pde_module_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,steps,iters,k", [(34, 4, 10, 3), (33, 3, 12, 12), (70, 2, 50, 10), (40, 5, 7, 1)])
def test_ldc_matches_operator_composition(n, steps, iters, k):
    s = P.FractionalStepLDC(n=n, Re=100.0, jacobi_iters=iters, jacobi_per_pass=k, dt=2e-3)
    rng = np.random.default_rng(n)
    u0 = (0.1 * rng.standard_normal(tuple(s.u.shape))).astype(np.float32)
    p0 = (0.1 * rng.standard_normal(tuple(s.p.shape))).astype(np.float32)
    s.u.copy_(torch.from_numpy(u0))
    s.p.copy_(torch.from_numpy(p0))
    s.step(steps, residuals=True)
    G = fdm.exterior_groups(u0.shape, 1)
    ug = [dict(ids=G["ALL"], type=1, value=0.0, comps=(0, 1)), dict(ids=G["+Y"], type=1, value=1.0, comps=(0,))]
    pg = [dict(ids=G["ALL"], type=2, value=0.0, comps=(0,))]
    u, p = u0, p0
    for _ in range(steps):
        u, p = fdm.ldc_step(u, p, ug, pg, s.dx, 1, s.nu, s.dt, iters)
    assert np.array_equal(s.u.cpu().numpy(), u)
    assert np.array_equal(s.p.cpu().numpy(), p)
    r = s.residuals.cpu().numpy()[:steps]
    assert np.all(np.isfinite(r)) and np.all(r >= 0)


def test_ldc_lid_drives_a_vortex():
    s = P.FractionalStepLDC(n=33, Re=100.0, jacobi_iters=50)
    s.step(400)
    u = s.u.cpu().numpy()[:, :, 0, :]
    mid = u.shape[0] // 2
    col = u[mid, 1:-1, 0]  # u along the vertical centre line, y from 0 to 1
    assert abs(col[-1] - 1.0) < 1e-2              # lid node (reset by the next step's boundary fill)
    assert col[-3] > 0.1                           # fluid dragged by the lid near the top
    assert col[len(col) // 4] < 0.0                # return flow in the lower half


@pytest.mark.parametrize("n,slabs,iters,k,steps", [(60, 2, 23, 5, 3), (75, 3, 12, 4, 2), (40, 1, 10, 3, 2)])
def test_slabs_match_whole_domain(n, slabs, iters, k, steps):
    """The cavity split into slabs along X (halo rows filled between phases, as the
    multi-GPU path does across ranks) is bit-identical to the whole-domain rollout."""
    from pde_module_b200.time_step.fractional_step import LDCSlab, slab_rows, ldc_slab_steps
    from pde_module_b200.distributed import exchange_local_slabs
    whole = P.FractionalStepLDC(n=n, Re=100.0, jacobi_iters=iters, jacobi_per_pass=k)
    whole.step(steps)
    halo = k + 1
    parts = [LDCSlab(r, n=n, Re=100.0, jacobi_iters=iters, jacobi_per_pass=k)
             for r in slab_rows(n + 2, slabs, halo)]
    ldc_slab_steps(parts, steps, lambda fields: exchange_local_slabs(fields, halo))
    torch.cuda.synchronize()
    for s in parts:
        rows = slice(s.own_lo, s.own_hi)
        assert torch.equal(s.u[s.owned], whole.u[rows]), (s.own_lo, s.own_hi)
        assert torch.equal(s.p[s.owned], whole.p[rows]), (s.own_lo, s.own_hi)


@pytest.mark.parametrize("n,g", [(15, 1), (31, 1), (63, 1), (127, 1), (14, 2), (62, 2), (29, 3), (20, 16)])
def test_ldc_tiles_of_ghosts_alone(n, g):
    """Velocity tiles (16 rows, 64 columns) that begin at the high ghosts or end at the low
    ones: a ghost's partner lies two cells inside, beyond the tile's neighbours."""
    s = P.FractionalStepLDC(n=n, Re=100.0, jacobi_iters=6, dt=1e-3 / n, ghost_cells=g)
    rng = np.random.default_rng(n)
    u = (0.1 * rng.standard_normal(tuple(s.u.shape))).astype(np.float32)
    p = (0.1 * rng.standard_normal(tuple(s.p.shape))).astype(np.float32)
    s.u.copy_(torch.from_numpy(u))
    s.p.copy_(torch.from_numpy(p))
    s.step(2)
    G = fdm.exterior_groups(u.shape, g)
    ug = [dict(ids=G["ALL"], type=1, value=0.0, comps=(0, 1)), dict(ids=G["+Y"], type=1, value=1.0, comps=(0,))]
    pg = [dict(ids=G["ALL"], type=2, value=0.0, comps=(0,))]
    for _ in range(2):
        u, p = fdm.ldc_step(u, p, ug, pg, s.dx, g, s.nu, s.dt, 6)
    assert np.array_equal(s.u.cpu().numpy(), u)
    assert np.array_equal(s.p.cpu().numpy(), p)


@pytest.mark.parametrize("n,cut", [(48, 33), (64, 33), (62, 31)])
def test_slab_of_one_row_more_than_its_tiles(n, cut):
    """The last slab owns 17 or 33 rows: its last velocity tile is the ghost row."""
    from pde_module_b200.time_step.fractional_step import LDCSlab, ldc_slab_steps
    from pde_module_b200.distributed import exchange_local_slabs
    X, halo = n + 2, 5
    whole = P.FractionalStepLDC(n=n, Re=100.0, jacobi_iters=8, jacobi_per_pass=4, dt=1e-3)
    whole.u.copy_(torch.rand(whole.u.shape, generator=torch.Generator().manual_seed(n)))
    parts = [LDCSlab(r, n=n, Re=100.0, jacobi_iters=8, jacobi_per_pass=4, dt=1e-3)
             for r in [(0, cut, 0, cut + halo), (cut, X, cut - halo, X)]]
    for s in parts:
        s.u.copy_(whole.u[s.held_lo:s.held_hi])
    whole.step(2)
    ldc_slab_steps(parts, 2, lambda fields: exchange_local_slabs(fields, halo))
    for s in parts:
        rows = slice(s.own_lo, s.own_hi)
        assert torch.equal(s.u_star[s.owned], whole._u_star[rows]), (s.own_lo, s.own_hi)
        assert torch.equal(s.u[s.owned], whole.u[rows]), (s.own_lo, s.own_hi)
        assert torch.equal(s.p[s.owned], whole.p[rows]), (s.own_lo, s.own_hi)
