"""Lines without a tensor map are described by tiles of 32 lines, as the
others are, whatever number of them a block takes: a batch is created with as
few descriptors.  The sizes leave whole and partial blocks of a tile."""
import re

import numpy as np
import pytest

from test_gpu_diffusion import O2, TOL, both_grids, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(300, 64, 1), (301, 41, 1), (39, 300, 1), (8, 257, 5), (265, 33, 3), (71, 9, 260)])
def test_tiles_of_long_lines(ctx, pcg, po, nx, ny, nz):
    from pcg import workloads
    g, subs, og, osubs = both_grids(pcg, po, nx, ny, nz, [O2])
    none = np.zeros(0)
    inst = workloads.instance(g, [O2], np.zeros((0, 3), np.float32), np.zeros(0, np.float32), 10.0, 0.4, 1.25, sec=none,
                              upt=none, sat=none, two_d=nz == 1)
    inst.density = np.random.default_rng(nx).uniform(0.0, 40.0, nx * ny * nz).astype(np.float32)
    b = pcg.Batch(ctx, [inst], autotune=False)
    text = b.describe()
    rows, cols = -(-ny * nz // 32), -(-nx // 32)
    want = {"x": rows if nx > 252 else 0, "y": cols * nz if ny > 256 else 0, "z": cols * ny if nz > 256 else 0}
    for axis, tiles in want.items():
        got = re.findall(axis + r":warp-lines\(,?tiles=(\d+)", text)
        assert got == ([str(tiles)] if tiles else []), text
    b.step(2)
    ref = inst.density.copy()
    for _ in range(2):
        po.sweeps(ref, og, osubs)
        po.dirichlet(ref, og, osubs)
    assert rel_err(b.density(0), ref) <= TOL
    b.close()
