"""The force pass stops at the distance past which both force terms are
exact zeros.  With diagnostics it walks the whole interaction distance, so
both must give the same bits, also for radii, adhesion reaches and strengths
that leave no such distance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cells(pcg, n, seed, side):
    from pcg import workloads
    rng = np.random.default_rng(seed)
    grid = pcg.make_grid(side, side, side, 1, dx=20.0, dt=0.01)
    pos = rng.uniform(0, side * 20.0, (n, 3)).astype(np.float32)
    radius = np.clip(rng.normal(8.4, 0.5, n), 5.0, 12.0).astype(np.float32)
    soa = workloads.make_soa(pos, radius, 10.0, 0.4, 1.25, grid)
    return grid, soa, rng


def _edit(pcg, case, f, n, rng):
    some = rng.random(n) < 0.02
    if case == "mixed_radii":
        f[pcg.F_RADIUS] = rng.uniform(0.0, 30.0, n)
    elif case == "zero_radius":
        f[pcg.F_RADIUS][:] = 0.0
    elif case == "negative_radius":
        f[pcg.F_RADIUS][some] = -9.0
    elif case == "nan_radius":
        f[pcg.F_RADIUS][some] = np.nan
    elif case == "inf_radius":
        f[pcg.F_RADIUS][some] = np.inf
    elif case == "relmax":
        f[pcg.F_REL_MAX_ADH] = rng.choice([-1.0, -0.0, 0.0, 0.5, 1.0, 1.25, 4.0, np.inf, np.nan], n)
    elif case == "strengths":
        f[pcg.F_REPULSION][some] = rng.choice([-1.0, 0.0, 1e38, np.inf, np.nan], int(some.sum()))
        f[pcg.F_ADHESION][:] = rng.choice([0.0, 1.0, 3e38], n)


@pytest.mark.parametrize("case", ["plain", "mixed_radii", "zero_radius", "negative_radius", "nan_radius", "inf_radius",
                                  "relmax", "strengths"])
def test_reach_keeps_the_bits(ctx, pcg, case):
    n, side = 3000, 10
    grid, soa, rng = _cells(pcg, n, 77, side)
    _edit(pcg, case, soa.reshape(pcg.NUM_FIELDS, n), n, rng)
    L = side * 20.0
    mech = pcg.mech_params_for_domain(0.0, L, 0.0, L, 0.0, L, False)
    out = []
    for diag in (False, True):
        cells = pcg.Cells(ctx, n, 1)
        cells.upload(soa, n, n)
        m = pcg.CellMechanics(ctx, mech, (0.0, 0.0, 0.0), n)
        m.set_diagnostics(diag)
        m.computeForces(cells)
        got = cells.download().reshape(pcg.NUM_FIELDS, -1)
        out.append(got[[pcg.F_VEL_X, pcg.F_VEL_Y, pcg.F_VEL_Z, pcg.F_PRESSURE]])
        if diag:
            assert m.neighbor_stats(n)[0].sum() > n   # every neighbour within the distance, still counted
        m.close()
        cells.close()
    a, b = out
    assert np.array_equal(np.isnan(a), np.isnan(b))
    ok = ~np.isnan(a)
    assert np.array_equal(a[ok].view(np.uint32), b[ok].view(np.uint32))


def test_reach_is_per_instance(ctx, pcg):
    """One instance of large cells beside one of small ones in a batch (their
    cells share blocks): each gets the bits it gets alone."""
    from pcg import workloads
    insts = []
    for k, (r, n) in enumerate(((8.4, 150), (14.0, 90), (2.0, 333))):
        rng = np.random.default_rng(k)
        grid = pcg.make_grid(8, 8, 8, 1, dx=20.0, dt=0.01)
        pos = rng.uniform(0, 160.0, (n, 3)).astype(np.float32)
        insts.append(workloads.instance(grid, [(1e5, 0.1, True, 38.0)], pos, np.full(n, r, np.float32), 10.0, 0.4, 1.25,
                                        sec=np.zeros(n), upt=np.full(n, 10.0), sat=np.zeros(n), two_d=False))
    def run(group):
        b = pcg.Batch(ctx, group, autotune=False)
        b.step(10)
        out = [b.cells(i) for i in range(len(group))]
        b.close()
        return out
    together = run(insts)
    for i, inst in enumerate(insts):
        assert np.array_equal(run([inst])[0].view(np.uint32), together[i].view(np.uint32)), i
