"""Lines solved from both ends, at the lengths where the halves change shape
(no interior node in the right half, every remainder of the last chunk, one
chunk more or less) and with couplings that settle in a few chunks, late, or
never: planes and tiles against the FP64 oracle, and against each other bit
for bit."""
import numpy as np
import pytest

from test_gpu_diffusion import TOL, both_grids, rel_err

pytestmark = pytest.mark.gpu

# D dt / dx^2 = 0.025, 2.5 and 250: g settles at once, after ~14 positions, never
SUBS = [(1e3, 0.5, True, 7.0), (1e5, 0.1, True, 38.0), (1e7, 0.01, False, 0.0)]


@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 19, 20, 33, 63, 64, 65, 130, 161,
                               236, 252])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_every_shape_of_halves(ctx, pcg, po, n, axis):
    shape = [5, 6, 4]
    shape[axis] = n
    nx, ny, nz = shape
    g, subs, og, osubs = both_grids(pcg, po, nx, ny, nz, SUBS)
    d0 = np.random.default_rng(100 * n + axis).uniform(0.0, 40.0, 3 * nx * ny * nz).astype(np.float32)
    ref = d0.copy()
    for _ in range(2):
        po.sweeps(ref, og, osubs)
        po.dirichlet(ref, og, osubs)
    mech = pcg.mech_params_for_domain(0, 60.0, 0, 60.0, 0, 60.0, False)
    got = []
    for planes in (True, False):
        b = pcg.Batch(ctx, [pcg.Instance(g, subs, mech, 0.1, density=d0)], autotune=False, planes=planes)
        b.step(2)
        got.append(b.density(0))
        b.close()
    assert rel_err(got[0], ref) <= TOL
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
