"""Cells that only take up (the secretion kernel's side-by-side path) against
IEEE FP64 arithmetic, bit for bit: one to four substrates, crowded voxels,
fields at zero, denormal and huge values, and rates that take the divisor out
of the quotient's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 2, 3, 4])
@pytest.mark.parametrize("wild", [False, True], ids=["plain", "wild"])
def test_uptake_is_ieee(ctx, pcg, S, wild):
    from pcg import workloads
    rng = np.random.default_rng(10 * S + wild)
    side, n = 9, 4000
    nv = side ** 3
    grid = pcg.make_grid(side, side, side, S, dx=20.0, dt=0.01)
    pos = rng.uniform(0, side * 20.0, (n, 3)).astype(np.float32)
    pos[: n // 4] = 5.0   # a thousand cells in one voxel
    soa = workloads.make_soa(pos, rng.uniform(5, 12, n).astype(np.float32), 10.0, 0.4, 1.25, grid)
    upt = rng.uniform(0, 50, (n, S))
    dens = rng.uniform(0, 40, (S, nv)).astype(np.float32)
    dens[:, rng.random(nv) < 0.2] = 0.0
    if wild:
        upt[rng.random((n, S)) < 0.02] = 1e90
        upt[rng.random((n, S)) < 0.02] = -1e75
        upt[rng.random((n, S)) < 0.01] = np.inf
        dens[:, rng.random(nv) < 0.1] = np.float32(1e-42)
        dens[:, rng.random(nv) < 0.1] = np.float32(3e38)
    me = pcg.Microenvironment(ctx, grid, pcg.make_substrates([(1e5, 0.1, True, 38.0)] * S))
    me.setDensityAll(dens)
    cells = pcg.Cells(ctx, n, S)
    cells.upload(soa, n, n)
    cells.set_secretion(None, upt.ravel(), None, None)
    me.applySecretion(cells, 0.01)
    got = me.densityBuffer().reshape(S, nv)
    vox = soa[26 * n:27 * n].view(np.uint32)
    ic = 0.01 * soa[11 * n:12 * n].astype(np.float64) / (20.0 * 20.0 * 20.0)
    ref = dens.copy()
    with np.errstate(all="ignore"):
        for c in range(n):
            rho = (ref[:, vox[c]].astype(np.float64) + 0.0) / (1.0 + ic[c] * (0.0 + upt[c]))
            ref[:, vox[c]] = np.where(rho < 0, 0.0, rho).astype(np.float32)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    ok = ~np.isnan(ref)
    assert np.array_equal(got[ok].view(np.uint32), ref[ok].view(np.uint32))
    cells.close()
    me.close()
