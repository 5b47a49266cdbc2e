"""Steps launched one after another without a wait between them: kernels of
later steps must not hold up the running ones.  A step of 100^3 voxels takes
1.0 to 1.4 times that of 90^3 (1.37 times the voxels, both under one wave of
planes); with kernels of several later steps waiting on the SMs, which the
smaller one still had room for, it took 2.2 times."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _step_seconds(ctx, pcg, side):
    grid = pcg.make_grid(side, side, side, 1, dx=20.0, dt=0.01)
    me = pcg.Microenvironment(ctx, grid, pcg.make_substrates([(1e5, 0.1, True, 38.0)]))
    me.fill(np.array([38.0], np.float32))
    best = 1e9
    for _ in range(7):
        ctx.sync()
        t = time.perf_counter()
        for _ in range(400):
            me.simulateDiffusionDecay(1)
        ctx.sync()
        best = min(best, (time.perf_counter() - t) / 400)
    me.close()
    return best


def test_steps_in_flight_do_not_hold_each_other_up(ctx, pcg):
    assert _step_seconds(ctx, pcg, 100) < 1.8 * _step_seconds(ctx, pcg, 90)
