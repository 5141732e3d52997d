"""The windowed element chase at its edges: orders of one to a few bands
(every op clipped, fewer sweeps than a group), and one past a multiple of the
group and of the window, in double-float and FP64, bands 16 and 32.  The band of
width ``tile`` goes straight to the window kernel for tiles 16 and 32, so the
whole call is compared with LAPACK (tolerances of the pipeline tests: FP64 1e-12,
FP32 class 1e-5, relative to the largest singular value)."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,mode,tol", [(np.float32, None, 1e-5), (np.float64, None, 1e-12),
                                         (np.float64, "fp64x2", 1e-12)])
@pytest.mark.parametrize("tile,tiles", [(16, 1), (16, 2), (16, 3), (16, 9), (16, 17), (32, 1), (32, 2), (32, 7)])
def test_window_chase_edges(avs_mod, dt, mode, tol, tile, tiles):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = tile * tiles
    a = np.random.default_rng(1000 * tile + tiles).standard_normal((n, n)).astype(dt)
    got = avs_mod.my_CU_svdval(avs_mod.to_device(a), tile, precision=mode).cpu().numpy().astype(np.float64)
    ref = sl.svdvals(a.astype(np.float64))
    assert np.max(np.abs(got - ref)) <= tol * ref[0]


@pytest.mark.parametrize("rank", [0, 1, 20])
def test_window_chase_zero_reflectors(avs_mod, rank):
    """Low rank: columns and rows that are exactly zero below the pivot give identity reflectors."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 80
    a = np.zeros((n, n))
    a[:rank, :rank] = np.random.default_rng(rank).standard_normal((rank, rank))
    got = avs_mod.my_CU_svdval(avs_mod.to_device(a), 16).cpu().numpy()
    ref = sl.svdvals(a)
    assert np.max(np.abs(got - ref)) <= 1e-12 * max(ref[0], 1.0)
