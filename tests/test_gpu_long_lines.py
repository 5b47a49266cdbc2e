"""Lines past the tensor boxes (one warp per line) against the FP64 oracle,
at the edges of the kernel's segment sizes: the largest line of each number
of positions per lane, one more, and several segments."""
import numpy as np
import pytest

from test_gpu_diffusion import O2, TOL, both_grids, rel_err

pytestmark = pytest.mark.gpu

# slowly decaying coupling too: D dt / dx^2 = 25, g close to 1
SUBS = [O2, (1e6, 0.01, False, 0.0)]


@pytest.mark.parametrize("shape", [(253, 9, 1), (384, 3, 1), (385, 8, 1), (512, 2, 1), (513, 17, 1), (768, 3, 1),
                                   (769, 5, 1), (1024, 3, 1), (1025, 9, 1), (2049, 4, 1), (7, 257, 1), (9, 1025, 1),
                                   (17, 2050, 1), (3, 5, 385), (257, 5, 6), (260, 300, 1)],
                         ids=lambda s: "x".join(map(str, s)))
def test_long_lines_match_oracle(ctx, pcg, po, shape):
    nx, ny, nz = shape
    g, subs, og, osubs = both_grids(pcg, po, nx, ny, nz, SUBS)
    d0 = np.random.default_rng(nx + ny + nz).uniform(0.0, 40.0, 2 * nx * ny * nz).astype(np.float32)
    me = pcg.Microenvironment(ctx, g, subs)
    me.setDensityAll(d0)
    ref = d0.copy()
    for k in range(3):
        me.step(None, 1)
        po.sweeps(ref, og, osubs)
        po.dirichlet(ref, og, osubs)
        assert rel_err(me.densityBuffer(), ref) <= TOL, k
    me.close()
