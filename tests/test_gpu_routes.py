"""Which kernels serve a call, by its launches: a single 2-D simulation's
sub-steps go into one launch only where there are few cells for the number of
sub-steps (else a plane pass and a secretion each), and the secretion order
of one simulation into one cluster up to 32768 cells.  What the fused launch
reads of the cells is what they are at the call: none secreting after all did,
voxels uploaded between calls; calls longer than one launch (256 sub-steps);
the bounded wait's way out."""
import numpy as np
import pytest

from test_gpu_failures import PCG_ERR_DEVICE
from test_gpu_steps_2d import _instance

pytestmark = pytest.mark.gpu


def _objects(ctx, pcg, inst):
    me = pcg.Microenvironment(ctx, inst.grid, inst.substrates)
    me.setDensityAll(inst.density)
    cells = pcg.Cells(ctx, inst.n_cells, inst.grid.n_substrates)
    cells.upload(inst.soa, inst.n_cells, inst.soa_max)
    cells.set_secretion(*inst.rates, active=inst.active)
    return me, cells


def _launches(ctx, f):
    before = ctx.launches
    f()
    return ctx.launches - before


@pytest.mark.parametrize("n,steps,fused", [(128, 1, True), (129, 1, False), (4096, 1, False), (1024, 2, True),
                                           (1025, 2, False), (2048, 3, True), (2049, 3, False), (3072, 4, True),
                                           (3073, 4, False), (4096, 5, True), (4097, 5, False), (4096, 256, True)])
def test_fused_steps_by_cells_and_sub_steps(ctx, pcg, n, steps, fused):
    me, cells = _objects(ctx, pcg, _instance(pcg, 50, 50, 2, n, n))
    me.step(cells, 1)   # builds the order
    assert _launches(ctx, lambda: me.step(cells, steps)) == (1 if fused else 2 * steps)
    assert _launches(ctx, lambda: me.step(None, steps)) == 1
    cells.close()
    me.close()


@pytest.mark.parametrize("n,cluster", [(1, True), (32768, True), (32769, False)])
def test_order_of_one_simulation(ctx, pcg, n, cluster):
    me, cells = _objects(ctx, pcg, _instance(pcg, 50, 50, 1, n, n))
    # constants, order and their permutation, secretion
    k = _launches(ctx, lambda: me.applySecretion(cells, 0.01))
    assert k == 4 if cluster else k > 4
    cells.close()
    me.close()


def test_fused_steps_read_the_cells_of_the_call(ctx, pcg):
    inst = _instance(pcg, 40, 31, 2, 700, 5)
    moved = inst.soa.copy()
    v = moved[pcg.F_VOXEL_IDX * inst.soa_max:][:700].view(np.uint32)
    v[:] = v[::-1] // 7   # other voxels, fewer runs
    out = []
    for fused in (True, False):
        me, cells = _objects(ctx, pcg, inst)
        # 700 cells take single sub-steps as a plane pass and a secretion
        go = (lambda k: me.step(cells, k)) if fused else (lambda k: [me.step(cells, 1) for _ in range(k)])
        got = []
        go(7)
        got.append(me.densityBuffer())
        cells.set_secretion(*inst.rates, active=np.zeros(700, np.uint8))   # none secretes
        go(3)
        got.append(me.densityBuffer())
        cells.set_secretion(*inst.rates, active=inst.active)
        cells.upload_fields(pcg.F_VOXEL_IDX, 1, moved, inst.soa_max)
        go(7)
        got.append(me.densityBuffer())
        go(300)
        got.append(me.densityBuffer())
        out.append(got)
        cells.close()
        me.close()
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), k


def test_fused_steps_report_a_wait_that_ran_out(ctx, pcg):
    inst = _instance(pcg, 50, 50, 1, 500, 9)
    me, cells = _objects(ctx, pcg, inst)
    me.step(cells, 10)
    ref = me.densityBuffer()
    L = pcg.lib()
    ctx.check(L.pcg_debug_give_up_waits(ctx.h, 1))
    try:
        assert _launches(ctx, lambda: me.step(cells, 10)) == 1
        st = L.pcg_sync(ctx.h)
    finally:
        ctx.check(L.pcg_debug_give_up_waits(ctx.h, 0))
    assert st == PCG_ERR_DEVICE
    assert b"wait limit" in L.pcg_last_error_string(ctx.h)
    assert L.pcg_sync(ctx.h) == 0
    me.setDensityAll(inst.density)
    me.step(cells, 10)
    assert np.array_equal(me.densityBuffer().view(np.uint32), ref.view(np.uint32))
    cells.close()
    me.close()
