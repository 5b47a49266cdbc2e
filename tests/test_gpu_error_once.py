"""A launch that CUDA refuses is reported by the call that made it and by no
later one.  Launches into the legacy stream are refused, on the host, while a
blocking stream is being captured."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CU_STREAM_LEGACY = 1
PCG_ERR_CUDA = 2   # include/pcg.h


def test_refused_launch_is_reported_once(pcg):
    ctx = pcg.Context(0, stream=CU_STREAM_LEGACY)
    grid = pcg.make_grid(40, 40, 1, 1, dx=20.0, dt=0.01)
    me = pcg.Microenvironment(ctx, grid, pcg.make_substrates([(1e5, 0.1, True, 38.0)]))
    me.setDensityAll(np.full(1600, 20.0, np.float32))
    me.step(None, 3)
    ref = me.computeGradients()
    L, cu = pcg.lib(), C.CDLL("libcuda.so.1")
    stream, graph = C.c_void_p(), C.c_void_p()
    assert cu.cuStreamCreate(C.byref(stream), 0) == 0
    assert cu.cuStreamBeginCapture_v2(stream, 0) == 0
    try:
        refused = [L.pcg_me_apply_dirichlet(me.h), L.pcg_me_diffuse(me.h, 1), L.pcg_me_step(me.h, None, 3)]
    finally:
        cu.cuStreamEndCapture(stream, C.byref(graph))
    if graph.value:
        assert cu.cuGraphDestroy(graph) == 0
    assert cu.cuStreamDestroy_v2(stream) == 0
    assert refused == [PCG_ERR_CUDA] * 3
    for a, b in zip(me.computeGradients(), ref):   # the next launch, by its own error alone
        assert np.array_equal(a, b)
    me.step(None, 3)
    me.close()
    ctx.sync()
    ctx.close()
