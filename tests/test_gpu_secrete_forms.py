"""Secretion against IEEE FP64 arithmetic, bit for bit, in both forms of the
kernel (few runs, many runs): one to five substrates, all terms or uptake
alone, crowded voxels, and operands that take the divisor or the dividend out
of the quotient's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("terms", ["uptake", "secretion", "all", "wild"])
@pytest.mark.parametrize("n", [4001, 760001])
def test_secretion_is_ieee(ctx, pcg, S, terms, n):
    from pcg import workloads
    rng = np.random.default_rng(n + 10 * S + len(terms))
    side = 13 if n < 10000 else 97
    nv = side ** 3
    grid = pcg.make_grid(side, side, side, S, dx=20.0, dt=0.01)
    pos = rng.uniform(0, side * 20.0, (n, 3)).astype(np.float32)
    pos[:50] = 5.0   # a crowded voxel
    soa = workloads.make_soa(pos, rng.uniform(5, 12, n).astype(np.float32), 10.0, 0.4, 1.25, grid)
    vox = soa[26 * n:27 * n].view(np.uint32)
    upt = rng.uniform(0, 50, (n, S))
    sec = rng.uniform(0, 5, (n, S)) if terms != "uptake" else np.zeros((n, S))
    sat = rng.uniform(0, 30, (n, S)) if terms != "uptake" else np.zeros((n, S))
    ne = rng.uniform(-20, 20, (n, S)) if terms in ("all", "wild") else np.zeros((n, S))
    dens = rng.uniform(0, 40, (S, nv)).astype(np.float32)
    if terms == "wild":
        upt[rng.random((n, S)) < 0.02] = 1e90
        upt[rng.random((n, S)) < 0.01] = np.inf
        ne[rng.random((n, S)) < 0.01] = 1e200
        ne[rng.random((n, S)) < 0.01] = -1e-300
        dens[:, rng.random(nv) < 0.1] = 0.0
        dens[:, rng.random(nv) < 0.1] = np.float32(1e-42)
        dens[:, rng.random(nv) < 0.1] = np.float32(3e38)
    me = pcg.Microenvironment(ctx, grid, pcg.make_substrates([(1e5, 0.1, True, 38.0)] * S))
    me.setDensityAll(dens)
    cells = pcg.Cells(ctx, n, S)
    cells.upload(soa, n, n)
    cells.set_secretion(sec.ravel(), upt.ravel(), sat.ravel(), ne.ravel())
    me.applySecretion(cells, 0.01)
    got = me.densityBuffer().reshape(S, nv)
    ref = dens.copy()
    with np.errstate(all="ignore"):
        V = 20.0 * 20.0 * 20.0
        ic = (0.01 * soa[11 * n:12 * n].astype(np.float64) / V)[:, None]
        c0, c1, c2 = 0.01 * ne / V, (ic * sec) * sat, 1.0 + ic * (sec + upt)
        # the k-th cell of every voxel at a time
        order = np.argsort(vox, kind="stable")
        head = np.r_[True, vox[order][1:] != vox[order][:-1]]
        first = np.flatnonzero(head)[np.cumsum(head) - 1]
        kth = np.arange(n) - first
        for k in range(int(kth.max()) + 1):
            c = order[kth == k]
            rho = ((ref[:, vox[c]].T.astype(np.float64) + c0[c]) + c1[c]) / c2[c]
            ref[:, vox[c]] = np.where(rho < 0, 0.0, rho).astype(np.float32).T
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    ok = ~np.isnan(ref)
    assert np.array_equal(got[ok].view(np.uint32), ref[ok].view(np.uint32))
    cells.close()
    me.close()
