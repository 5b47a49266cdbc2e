"""Several sub-steps of a 2-D simulation in one launch (pcg_me_step, the plane
and its cells' terms in shared memory) against the batch's passes, bit for
bit: sides at the edges of the solver classes, planes far from square, few
and many cells per voxel, export, secretion, uptake, inactive cells, fields
at zero, and operands that leave the side-by-side quotient's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _instance(pcg, nx, ny, S, n, seed, wild=False):
    from pcg import workloads
    rng = np.random.default_rng(seed)
    grid = pcg.make_grid(nx, ny, 1, S, dx=20.0, dt=0.01, z_min=-10.0)
    subs = [(1e5, 0.1, True, 38.0), (2e3, 0.4, False, 0.0), (3e4, 0.0, True, 0.0)][:S]
    pos = np.zeros((n, 3), np.float32)
    pos[:, 0] = rng.uniform(0, nx * 20.0, n)
    pos[:, 1] = rng.uniform(0, min(ny, 5 + n // 40) * 20.0, n)   # crowded: many cells in a voxel
    k = n * S
    sec, upt = rng.uniform(0, 5, k), rng.uniform(0, 20, k)
    ne = np.where(rng.random(k) < 0.3, rng.uniform(-200, 200, k), 0.0)
    sat = rng.uniform(0, 40, k)
    if wild:
        upt[rng.random(k) < 0.05] = -1e80
        upt[rng.random(k) < 0.05] = 1e90
        ne[rng.random(k) < 0.05] = 1e200
        sat[rng.random(k) < 0.05] = np.inf
    inst = workloads.instance(grid, subs, pos, np.full(n, 8.4, np.float32), 10.0, 0.4, 1.25, sec=sec, upt=upt, sat=sat,
                              ne=ne)
    inst.active = (rng.random(n) < 0.9).astype(np.uint8)
    inst.density = np.where(rng.random(S * nx * ny) < 0.3, 0.0, rng.uniform(0, 40, S * nx * ny)).astype(np.float32)
    return inst


@pytest.mark.parametrize("nx,ny,S,n,wild", [(50, 50, 1, 500, False), (13, 13, 2, 60, False), (64, 64, 3, 4096, False),
                                            (64, 12, 1, 1, False), (7, 33, 2, 40, False), (65, 64, 1, 900, False),
                                            (128, 40, 2, 2000, False), (128, 128, 1, 3000, False),
                                            (129, 20, 2, 300, False), (236, 40, 1, 1500, False), (20, 252, 1, 700, False),
                                            (64, 64, 1, 4097, False), (40, 31, 2, 700, True)],
                         ids=lambda v: str(v))
def test_steps_in_one_launch(ctx, pcg, nx, ny, S, n, wild):
    inst = _instance(pcg, nx, ny, S, n, nx * 1000 + ny, wild)
    steps = 7   # no mechanics step in the batch
    b = pcg.Batch(ctx, [inst], autotune=False)
    b.step(steps)
    ref = b.density(0)
    b.close()
    me = pcg.Microenvironment(ctx, inst.grid, inst.substrates)
    cells = pcg.Cells(ctx, n, S)
    cells.upload(inst.soa, n, inst.soa_max)
    cells.set_secretion(*inst.rates, active=inst.active)
    for calls in ([steps], [1] * steps, [3, 4]):
        me.setDensityAll(inst.density)
        for k in calls:
            me.step(cells, k)
        got = me.densityBuffer()
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        ok = ~np.isnan(ref)
        assert np.array_equal(got[ok].view(np.uint32), ref[ok].view(np.uint32)), calls
    for x in (cells, me):
        x.close()
