"""z planes cut into strips of columns (large planes, of which an SM holds few)
against the FP64 oracle, faces and ragged last strips included."""
import numpy as np
import pytest

from test_gpu_diffusion import O2, TOL, both_grids, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(150, 150, 150), (149, 152, 140), (131, 151, 150)], ids=lambda s: "x".join(map(str, s)))
def test_strips_match_oracle(ctx, pcg, po, shape):
    nx, ny, nz = shape
    subs_p = [O2, (5e3, 0.2, False, 0.0)]
    g, subs, og, osubs = both_grids(pcg, po, nx, ny, nz, subs_p)
    d0 = np.random.default_rng(nx).uniform(0.0, 40.0, 2 * nx * ny * nz).astype(np.float32)
    inst = pcg.Instance(g, subs, pcg.mech_params_for_domain(0, 60.0, 0, 60.0, 0, 60.0, False), 0.1, density=d0)
    b = pcg.Batch(ctx, [inst], autotune=False)
    jobs = [int(w.split("jobs=")[1].split(",")[0]) for w in b.describe().split() if w.startswith("z:xz-planes")]
    assert sum(jobs) > 2 * ny   # more jobs than planes: strips
    b.step(1)
    got = b.density(0)
    b.close()
    po.sweeps(d0, og, osubs)
    po.dirichlet(d0, og, osubs)
    assert rel_err(got, d0) <= TOL
