"""FP64 columns whose squares underflow (entries around 1e-165 and below): the
reflectors cannot be formed, so the calls fail with the non-finite status instead of
returning values of an unreduced matrix.  Entries of 1e-140 are still factored, and
exact zeros are no reason to refuse."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu

NONFINITE = 4  # AVS_ERR_NONFINITE


def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("scale", [1e-165, 1e-200, 1e-300])
@pytest.mark.parametrize("tile,tiles", [(16, 3), (32, 1), (64, 2), (128, 2), (256, 2)])
def test_underflowing_columns_are_refused(avs_mod, tile, tiles, scale):
    cuda()
    a = np.random.default_rng(tile).standard_normal((tile * tiles, tile * tiles)) * scale
    for call in (avs_mod.my_CU_svdval, avs_mod.tiled_QR):
        with pytest.raises(avs_mod.AvsError) as e:
            call(avs_mod.to_device(a), tile)
        assert e.value.status == NONFINITE


@pytest.mark.parametrize("tile,tiles", [(16, 3), (64, 2), (128, 2)])
def test_small_and_zero_columns_are_not(avs_mod, tile, tiles):
    cuda()
    n = tile * tiles
    a = np.random.default_rng(tile).standard_normal((n, n)) * 1e-140
    a[:, 3] = 0.0
    got = avs_mod.my_CU_svdval(avs_mod.to_device(a), tile).cpu().numpy()
    ref = sl.svdvals(a * 1e140)
    assert np.max(np.abs(got * 1e140 - ref)) <= 1e-12 * ref[0]
    assert np.all(avs_mod.my_CU_svdval(avs_mod.to_device(np.zeros((n, n))), tile).cpu().numpy() == 0.0)
