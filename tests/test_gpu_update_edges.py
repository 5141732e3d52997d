"""The SIMT trailing updates at the edges of their split: ragged strips (orders
that are not a multiple of the strip width), few and many tiles, against LAPACK
on the whole call (FP64 1e-12, FP32 class 1e-5 of the largest value); and the
choices that must not change a value: one tile per CTA or all of them (a single
call and a batch of the same matrices), and a counter per block or per strip (in
core and out of core)."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu


def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("dt,mode,tol", [(np.float32, None, 1e-5), (np.float64, None, 1e-12),
                                         (np.float64, "fp64x2", 1e-12)])
@pytest.mark.parametrize("tile,tiles", [(16, 7), (16, 23), (32, 2), (32, 9), (64, 2), (64, 7), (128, 2), (128, 5),
                                        (256, 2)])
def test_update_edges(avs_mod, dt, mode, tol, tile, tiles):
    cuda()
    n = tile * tiles
    a = np.random.default_rng(3 * tile + tiles).standard_normal((n, n)).astype(dt)
    got = avs_mod.my_CU_svdval(avs_mod.to_device(a), tile, precision=mode).cpu().numpy().astype(np.float64)
    ref = sl.svdvals(a.astype(np.float64))
    assert np.max(np.abs(got - ref)) <= tol * ref[0]


@pytest.mark.parametrize("tile,n,count", [(32, 160, 110), (64, 320, 80), (64, 448, 50)])
def test_update_grouping_keeps_the_values(avs_mod, tile, n, count):
    torch = cuda()
    rng = np.random.default_rng(n)
    mats = [avs_mod.to_device(rng.standard_normal((n, n)).astype(np.float32)) for _ in range(4)]
    outs = avs_mod.svdvals_batched([mats[i % 4] for i in range(count)], tiles=tile)
    for i in range(4):
        single = avs_mod.my_CU_svdval(mats[i], tile)
        assert all(torch.equal(outs[q], single) for q in range(i, count, 4))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("tile,n", [(32, 480), (64, 704)])
def test_update_out_of_core_counters(avs_mod, dt, tile, n):
    cuda()
    a = np.asfortranarray(np.random.default_rng(n).standard_normal((n, n)).astype(dt))
    t = avs_mod.to_device(a)
    avs_mod.Blockbidiag(t, tile)
    h = a.copy(order="F")
    avs_mod.OOC_Bidiag(h, tile, device_bytes=6 * tile * n * h.itemsize + (1 << 20))
    assert np.array_equal(h, avs_mod.from_device(t))
