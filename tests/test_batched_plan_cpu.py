"""The progress words of a batched plan lie inside the work buffer.  The plan's
host side needs no GPU: everything but its block count is there when the upload
of the table fails for want of a device."""
import ctypes as C

import numpy as np
import pytest
import torch

from pde_module_b200 import _lib

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="plans into an address that is no device memory")

# narrow boxes are split where a side is not a multiple of the strip or the lane
THIN = [(150, 50), (200, 30), (300, 61), (661, 25), (25, 25), (1015, 25), (1000, 60), (28, 57), (126, 57)]


def _dirichlet(shape):
    grp = (_lib.PdeBCGroup * 1)()
    grp[0].type, grp[0].comp_mask, grp[0].face_mask = _lib.PDE_BC_DIRICHLET, 1, 0xF
    rules = _lib.PdeBCRules()
    grid = _lib.make_grid(shape, 1, 2, 0.1)
    assert _lib.lib().pde_bc_compile(grp, 1, C.byref(grid), 1, C.byref(rules)) == _lib.PDE_OK
    return rules


def _plan(kind, box, g, k, work_bytes=None, tile=(0, 0)):
    """(plan, work bytes asked for) of one grid with this box; None when the arguments are refused."""
    pad = g + (kind == _lib.PDE_BATCH_WAVE)
    desc = (_lib.PdeBatchGrid * 1)()
    d = desc[0]
    d.field, d.field_prev, d.scratch = 1 << 20, 2 << 20, 3 << 20
    d.shape[0], d.shape[1] = box[0] + 2 * pad, box[1] + 2 * pad
    d.dx, d.coef, d.dt = 0.1, 0.1, 0.1
    need = C.c_uint64(0)
    L = _lib.lib()
    assert L.pde_batch_work_bytes(desc, 1, *tile, C.byref(need)) == _lib.PDE_OK
    plan = _lib.PdeBatchPlan()
    rules = _dirichlet((box[0] + 2 * pad, box[1] + 2 * pad, 1))
    rc = L.pde_batch_plan(kind, desc, 1, g, 2, C.byref(rules), *tile, k, C.c_void_p(4 << 20),
                          need.value if work_bytes is None else work_bytes, C.byref(plan), None)
    if rc in (_lib.PDE_ERR_ARG, _lib.PDE_ERR_TOO_LARGE):
        return None
    assert rc == _lib.PDE_ERR_CUDA and plan.total_tiles > 0
    return plan, need.value


def _bytes(tiles):  # table of one grid, queue counter, progress words
    return 256 + 256 + 4 * tiles


@pytest.mark.parametrize("kind", [_lib.PDE_BATCH_HEAT, _lib.PDE_BATCH_WAVE])
@pytest.mark.parametrize("tile,depths", [((0, 0), range(0, 33)), ((20, 48), range(0, 21, 4)), ((40, 0), range(0, 13, 2)),
                                         ((0, 100), range(0, 33, 4))])
def test_progress_words_fit_the_work_buffer(kind, tile, depths):
    rng = np.random.default_rng(3)
    sides = [tuple(int(v) for v in rng.integers(8, 701, 2)) for _ in range(60)]
    register = 0
    for k in depths:
        for box in THIN + sides:
            made = _plan(kind, box, 1 + (box[0] & 1), k, tile=tile)
            if made:
                plan, need = made
                register += plan.register_tiles
                assert _bytes(plan.total_tiles) <= need, (box, k)
    assert register > (500 if tile == (0, 0) else 0)


def test_a_small_work_buffer_takes_the_shared_memory_tiles():
    """150 x 50 takes 8 register tiles; 5 x 1 shared-memory tiles of 32 x 64."""
    plan, _ = _plan(_lib.PDE_BATCH_HEAT, (150, 50), 1, 0)
    assert plan.register_tiles == 1 and plan.total_tiles == 8
    plan, _ = _plan(_lib.PDE_BATCH_HEAT, (150, 50), 1, 0, work_bytes=_bytes(7))
    assert plan.register_tiles == 0 and plan.total_tiles == 5
    assert _plan(_lib.PDE_BATCH_HEAT, (150, 50), 1, 0, work_bytes=_bytes(4)) is None
