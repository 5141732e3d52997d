"""The block stage in double-float (FP64 tiles with double-float stages): bands
64, 128 and 256 to 16 and 32, one tile to a few (no op past the first panel;
every op clipped; a last panel of one column), full and zero columns.  Values
against LAPACK within 1e-12 of the largest, the bound of this mode everywhere,
and against the one-stage chase of the same band."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu

ONE_STAGE, BAND32 = 4, 8


@pytest.mark.parametrize("flags", [0, BAND32])
@pytest.mark.parametrize("tile,tiles,rank", [(64, 1, None), (64, 2, None), (64, 5, 70), (128, 1, None), (128, 3, None),
                                             (128, 4, 129), (256, 1, None), (256, 3, None), (128, 2, 0)])
def test_double_float_block_stage(avs_mod, flags, tile, tiles, rank):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = tile * tiles
    rng = np.random.default_rng(100 * tile + tiles)
    a = rng.standard_normal((n, n))
    if rank is not None:
        a[rank:, :] = 0.0
        a[:, rank:] = 0.0
    call = lambda f: avs_mod.my_CU_svdval(avs_mod.to_device(a), tile, precision="fp64x2", flags=f).cpu().numpy()
    got = call(flags)
    ref = sl.svdvals(a)
    bound = 1e-12 * max(ref[0], 1.0)
    assert np.max(np.abs(got - ref)) <= bound
    assert np.max(np.abs(got - call(flags | ONE_STAGE))) <= 2 * bound
