"""Rows of the panel's diagonal blocks pass from role to role in tagged words of a
buffer that later stages overwrite: calls of other orders, tiles and types on the
same handle in between must not leave anything a later call takes for its own, so
the same matrix gives the same bits.  (The path without the buffer is out of core,
whose results are compared with these bit for bit in its own tests.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_panel_mailbox_reuse(avs_mod, tile, dt):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(tile)
    sizes = [5 * tile, 2 * tile, 3 * tile, 5 * tile]
    mats = [rng.standard_normal((n, n)).astype(dt) for n in sizes]

    def factor(a):
        d = avs_mod.to_device(a)
        avs_mod.tiled_QR(d, tile)
        torch.cuda.synchronize()
        return d.cpu().numpy()

    def values(a):
        return avs_mod.my_CU_svdval(avs_mod.to_device(a), tile).cpu().numpy()

    first = [(factor(a), values(a)) for a in mats]
    for i in (3, 1, 0, 2):
        assert np.array_equal(factor(mats[i]), first[i][0])
        assert np.array_equal(values(mats[i]), first[i][1])
