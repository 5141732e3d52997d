"""The stage-1 panel at the edges of its split: one, two and an odd number of
tiles for every tile size, in FP32, FP64 and double-float, against LAPACK on the
whole call (tolerances of the pipeline tests, relative to the largest singular
value), and the tau and R of a tiled QR of two tiles against the oracle's tile
kernels.  Inputs include columns that are exactly zero and a matrix scaled out of
FP32's range (FP64), which take the general branches of the reflector scalars."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu

MODES = [(np.float32, None, 1e-5), (np.float64, None, 1e-12), (np.float64, "fp64x2", 1e-12)]


def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("dt,mode,tol", MODES)
@pytest.mark.parametrize("tile,tiles", [(16, 5), (32, 1), (32, 3), (64, 1), (64, 3), (128, 1), (128, 3), (256, 1),
                                        (256, 3)])
def test_panel_edges(avs_mod, dt, mode, tol, tile, tiles):
    cuda()
    n = tile * tiles
    a = np.random.default_rng(tile + tiles).standard_normal((n, n)).astype(dt)
    a[:, n // 2] = 0.0
    got = avs_mod.my_CU_svdval(avs_mod.to_device(a), tile, precision=mode).cpu().numpy().astype(np.float64)
    ref = sl.svdvals(a.astype(np.float64))
    assert np.max(np.abs(got - ref)) <= tol * ref[0]


@pytest.mark.parametrize("scale", [1e-60, 1e60])
@pytest.mark.parametrize("tile", [16, 64])
def test_panel_fp64_range(avs_mod, scale, tile):
    """FP64 keeps FP64's exponent range (norms outside FP32's)."""
    cuda()
    n = 3 * tile
    a = np.random.default_rng(tile).standard_normal((n, n)) * scale
    got = avs_mod.my_CU_svdval(avs_mod.to_device(a), tile).cpu().numpy()
    ref = sl.svdvals(a)
    assert np.max(np.abs(got - ref)) <= 1e-12 * ref[0]


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("tile", [16, 32, 64, 128, 256])
def test_panel_two_tiles_vs_oracle(avs_mod, oracle_mod, dt, tile):
    cuda()
    a = np.random.default_rng(7 * tile).random((2 * tile, 2 * tile)).astype(dt)
    t = avs_mod.to_device(a)
    tau = avs_mod.tiled_QR(t, tile).cpu().numpy()
    f = avs_mod.from_device(t)
    f0, t0 = oracle_mod.geqrt(a[:tile, :tile])
    r1, v1, t1 = oracle_mod.tsqrt(f0, a[tile:, :tile])
    tol = 50 * np.finfo(dt).eps * tile
    assert np.max(np.abs(tau[:tile - 1] - t0[:tile - 1])) < tol
    assert np.max(np.abs(tau[tile:2 * tile] - t1)) < tol
    assert np.max(np.abs(np.triu(f[:tile, :tile]) - np.triu(r1))) < tol * np.max(np.abs(r1))
    assert np.max(np.abs(f[tile:, :tile] - v1)) < tol * np.max(np.abs(v1))
