"""The secretion order of one simulation built by one cluster, and just past
it: a voxel's cells act in ascending index, so uptake and secretion come out
as IEEE FP64 arithmetic in that order, bit for bit, over the sizes of its
tiles, one to three digit passes, cells outside the grid and inactive ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 2, 1), (41, 37, 29), (70, 66, 64)], ids=["1voxel", "1pass", "2pass", "3pass"])
@pytest.mark.parametrize("n", [1, 33, 1024, 1025, 8192, 8193, 16385, 32768, 32769])
def test_order_of_a_voxels_cells(ctx, pcg, dims, n):
    from pcg import workloads
    rng = np.random.default_rng(n + dims[0])
    S, nv = 2, int(np.prod(dims))
    grid = pcg.make_grid(*dims, S, dx=20.0, dt=0.01)
    pos = (rng.uniform(0, 20.0, (n, 3)) * np.asarray(dims)).astype(np.float32)
    pos[rng.random(n) < 0.02] = 5.0   # a crowded voxel
    soa = workloads.make_soa(pos, rng.uniform(5, 12, n).astype(np.float32), 10.0, 0.4, 1.25, grid)
    vox = soa[26 * n:27 * n].view(np.uint32)
    vox[rng.random(n) < 0.05] = nv + 7   # outside the grid: takes no part
    active = (rng.random(n) < 0.9).astype(np.uint8)
    sec, upt, sat = rng.uniform(0, 5, (n, S)), rng.uniform(0, 50, (n, S)), rng.uniform(0, 30, (n, S))
    dens = rng.uniform(0, 40, (S, nv)).astype(np.float32)
    me = pcg.Microenvironment(ctx, grid, pcg.make_substrates([(1e5, 0.1, True, 38.0)] * S))
    me.setDensityAll(dens)
    cells = pcg.Cells(ctx, n, S)
    cells.upload(soa, n, n)
    cells.set_secretion(sec.ravel(), upt.ravel(), sat.ravel(), None, active)
    me.applySecretion(cells, 0.01)
    got = me.densityBuffer().reshape(S, nv)
    ic = 0.01 * soa[11 * n:12 * n].astype(np.float64) / (20.0 * 20.0 * 20.0)
    c1 = (ic[:, None] * sec) * sat
    c2 = 1.0 + ic[:, None] * (sec + upt)
    ref = dens.copy()
    for c in np.flatnonzero((active != 0) & (vox < nv)):
        rho = (ref[:, vox[c]].astype(np.float64) + c1[c]) / c2[c]
        ref[:, vox[c]] = np.where(rho < 0, 0.0, rho).astype(np.float32)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    cells.close()
    me.close()
