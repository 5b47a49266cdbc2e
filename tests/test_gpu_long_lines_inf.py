"""An infinite density on a line past the tensor boxes (one warp per line,
the recurrences scanned over its lanes): every interior value of the line is
infinite with the same sign, as the FP64 oracle's walk leaves it, and never
NaN; another substrate keeps its values.  The infinite value lies beside
either end, inside the line, and at the edges of the lanes' and segments'
positions; in lines of one segment and of several."""
import numpy as np
import pytest

from test_gpu_diffusion import O2, TOL, both_grids, rel_err

pytestmark = pytest.mark.gpu

SUBS = [(2e3, 0.1, False, 0.0), O2]


@pytest.mark.parametrize("shape", [(253, 3, 1), (384, 9, 1), (701, 5, 1), (1030, 3, 1), (4, 300, 1), (3, 2050, 1),
                                   (5, 4, 257)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_infinite_value_stays_infinite(ctx, pcg, po, shape, value):
    nx, ny, nz = shape
    g, subs, og, osubs = both_grids(pcg, po, nx, ny, nz, SUBS)
    nv = nx * ny * nz
    axis = int(np.argmax(shape))
    n, step = shape[axis], (1, nx, nx * ny)[axis]
    start = sum(k * s for k, s in zip([0 if a == axis else shape[a] // 2 for a in range(3)], (1, nx, nx * ny)))
    me = pcg.Microenvironment(ctx, g, subs)
    for p in sorted({1, 11, 12, 23, n // 2, min(1023, n - 2), min(1024, n - 2), n - 2}):
        d0 = np.random.default_rng(p).uniform(0.0, 40.0, 2 * nv).astype(np.float32)
        d0[start + p * step] = value
        ref = d0.copy()
        po.sweeps(ref, og, osubs)
        me.setDensityAll(d0)
        me.simulateDiffusionDecay(1)
        got = me.densityBuffer()
        assert not np.isnan(ref).any() and np.isinf(ref).sum() >= n - 2
        assert np.array_equal(np.isposinf(got), np.isposinf(ref)), p
        assert np.array_equal(np.isneginf(got), np.isneginf(ref)), p
        ok = np.isfinite(ref)
        assert np.isfinite(got[ok]).all(), p
        assert rel_err(got[ok], ref[ok]) <= TOL, p
    me.close()
