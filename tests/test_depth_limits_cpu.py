"""A pass depth whose region does not fit in shared memory is refused, whichever
kernel would run: depths are checked on the host before the first call to the device."""
import ctypes as C

import pytest
import torch

from pde_module_b200 import _lib

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="passes addresses that are no device memory")


def _ptrs(n):
    return [C.c_void_p(1 << (20 + i)) for i in range(n)]


def _rules(shape, g, ncomp, typ):
    grp = (_lib.PdeBCGroup * 1)()
    grp[0].type, grp[0].comp_mask, grp[0].face_mask = typ, (1 << ncomp) - 1, 0xF
    rules = _lib.PdeBCRules()
    grid = _lib.make_grid(shape, g, 2, 0.1)
    assert _lib.lib().pde_bc_compile(grp, 1, C.byref(grid), ncomp, C.byref(rules)) == _lib.PDE_OK
    return rules


@pytest.mark.parametrize("side", [66, 258, 1026])
@pytest.mark.parametrize("k,nsteps,rc", [(100, 300, _lib.PDE_ERR_TOO_LARGE), (100, 16, _lib.PDE_ERR_CUDA),
                                         (16, 300, _lib.PDE_ERR_CUDA), (0, 300, _lib.PDE_ERR_CUDA)])
def test_heat_depth(side, k, nsteps, rc):
    shape = (side, side, 1)
    grid, rules = _lib.make_grid(shape, 1, 2, 0.1), _rules(shape, 1, 1, _lib.PDE_BC_DIRICHLET)
    assert _lib.lib().pde_heat_rollout(*_ptrs(3), C.byref(grid), 1, C.byref(rules), 1.0, 1e-4, nsteps, k, None) == rc


@pytest.mark.parametrize("n", [64, 256, 1024])
@pytest.mark.parametrize("k,iters,rc", [(100, 300, _lib.PDE_ERR_TOO_LARGE), (100, 16, _lib.PDE_ERR_CUDA),
                                        (12, 300, _lib.PDE_ERR_CUDA), (0, 300, _lib.PDE_ERR_CUDA)])
def test_cavity_depth(n, k, iters, rc):
    shape = (n + 2, n + 2, 1)
    grid = _lib.make_grid(shape, 1, 2, 1.0 / n)
    ru, rp = _rules(shape, 1, 2, _lib.PDE_BC_DIRICHLET), _rules(shape, 1, 1, _lib.PDE_BC_VON_NEUMANN)
    prm = _lib.PdeLDCParams(0.01, 1e-4, iters, k)
    L = _lib.lib()
    assert L.pde_ldc_rollout(*_ptrs(5), None, C.byref(grid), C.byref(ru), C.byref(rp), C.byref(prm), 1, None) == rc
    if k > iters or k == 0:
        return
    slab = _lib.PdeSlab(n + 2, 0, 0, n + 2)
    u, us, pin, pout, rhs = _ptrs(5)
    assert L.pde_ldc_slab_step(_lib.PDE_LDC_JACOBI, u, us, pin, pout, rhs, None, C.byref(grid), C.byref(slab),
                               C.byref(ru), C.byref(rp), C.byref(prm), k, 0, None) == rc
