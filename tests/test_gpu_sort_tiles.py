"""The static pair sort at the sizes where its tiles and the batches of rows
that a tile adds up begin and end: order and stability, few and many digits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 2048, 2049, 8193, 65537, 129 * 1024, 262143])
@pytest.mark.parametrize("bits", [3, 8, 9, 32])
def test_sort(ctx, pcg, n, bits):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    keys[: n // 3] = keys[0]
    kd = torch.from_numpy(keys.view(np.int32)).cuda()
    vd = torch.arange(n, dtype=torch.int32, device="cuda")
    ko, vo = torch.empty_like(kd), torch.empty_like(vd)
    ctx.check(pcg.lib().pcg_sort_pairs_static(ctx.h, None, None, None, None, 0, 32))   # set-up call
    torch.cuda.synchronize()
    ctx.check(pcg.lib().pcg_sort_pairs_static(ctx.h, kd.data_ptr(), vd.data_ptr(), ko.data_ptr(), vo.data_ptr(), n, bits))
    ctx.sync()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(vo.cpu().numpy().view(np.uint32), order.astype(np.uint32))
    assert np.array_equal(ko.cpu().numpy().view(np.uint32), keys[order])
