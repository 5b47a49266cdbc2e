"""The cell-start table at the sizes where its scan changes shape: one tile,
one block, tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (23, 89, 1), (32, 64, 1), (7, 31, 151), (32, 32, 32), (33, 32, 32)],
                         ids=lambda d: "x".join(map(str, d)))
def test_start_table(ctx, pcg, dims):
    n = 5000
    rng = np.random.default_rng(sum(dims))
    size = np.array(dims) * 30.0
    soa = np.zeros((pcg.NUM_FIELDS, n), np.float32)
    soa[:3] = (rng.uniform(0, 1, (n, 3)) ** 2 * size).astype(np.float32).T
    soa[pcg.F_RADIUS] = 8.0
    cells = pcg.Cells(ctx, n, 1)
    cells.upload(soa.ravel(), n, n)
    m = pcg.CellMechanics(ctx, pcg.MechanicsParams(0.1, 10.0, 0.4, 30.0, 30.0, *dims), (0.0, 0.0, 0.0), n)
    m.computeForces(cells)
    start, order = m.syncHashPointers(n)
    b = [np.clip(np.trunc(soa[a] / np.float32(30.0)).astype(np.int64), 0, dims[a] - 1) for a in range(3)]
    key = (b[2] * dims[1] + b[1]) * dims[0] + b[0]
    want = np.r_[0, np.cumsum(np.bincount(key, minlength=int(np.prod(dims))))]
    assert np.array_equal(start, want)
    assert np.array_equal(order, np.argsort(key, kind="stable"))
    m.close()
    cells.close()
