"""The two forms of the force pass (few cells, many cells) give the bits of
the pass with diagnostics, which always takes the second form: one cell, odd
sizes, both sides of the line between them, plane and volume, crowded rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LINE = 2 * 148 * 3 * 256


@pytest.mark.parametrize("n", [1, 255, 3001, LINE, LINE + 1])
@pytest.mark.parametrize("flat", [False, True], ids=["3d", "2d"])
def test_forms_agree(ctx, pcg, n, flat):
    from pcg import workloads
    rng = np.random.default_rng(n + flat)
    side = max(4, int((n / 2.0) ** (1 / 2 if flat else 1 / 3)))
    dims = (side, side, 1 if flat else side)
    L = side * 20.0
    grid = pcg.make_grid(*dims, 1, dx=20.0, dt=0.01)
    pos = (rng.uniform(0, 20.0, (n, 3)) * np.asarray(dims)).astype(np.float32)
    pos[: min(n, 300)] *= np.float32(20.0 / L)   # a crowded corner
    if flat:
        pos[:, 2] = 0.0
    soa = workloads.make_soa(pos, np.clip(rng.normal(8.4, 0.5, n), 5.0, 12.0).astype(np.float32), 10.0, 0.4, 1.25, grid)
    mech = pcg.mech_params_for_domain(0.0, L, 0.0, L, 0.0, 20.0 if flat else L, flat)
    out = []
    for diag in (False, True):
        cells = pcg.Cells(ctx, n, 1)
        cells.upload(soa, n, n)
        m = pcg.CellMechanics(ctx, mech, (0.0, 0.0, 0.0), n)
        m.set_diagnostics(diag)
        m.computeForces(cells)
        got = cells.download().reshape(pcg.NUM_FIELDS, -1)
        out.append(got[[pcg.F_VEL_X, pcg.F_VEL_Y, pcg.F_VEL_Z, pcg.F_PRESSURE]])
        m.close()
        cells.close()
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
