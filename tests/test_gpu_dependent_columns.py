"""Matrices with exactly or nearly dependent columns (all ones, low rank, sparse,
Hilbert): cancellation leaves columns some 1e-8 (FP32) or 1e-16 (FP64) of the ones
before them, again and again, down to the end of the type's range.  Such a column
counts as zero: the calls succeed, in core, in batches and out of core, with the
values of LAPACK (FP64 1e-12; the FP32 class, and double-float whose columns end
where FP32's range does, 1e-5 of the largest).  A matrix that is itself at the end
of the range is refused or right, never wrong with success."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu

MODES = [(np.float32, None, 1e-5), (np.float64, None, 1e-12), (np.float64, "fp64x2", 1e-5)]


def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def matrix(kind, n):
    rng = np.random.default_rng(7)
    if kind == "ones":
        return np.ones((n, n))
    if kind == "rank 3":
        return rng.standard_normal((n, 3)) @ rng.standard_normal((3, n))
    if kind == "sparse":
        return rng.standard_normal((n, n)) * (rng.random((n, n)) < 0.02)
    i = np.arange(n)
    return 1.0 / (i[:, None] + i[None] + 1.0)


@pytest.mark.parametrize("dt,mode,tol", MODES)
@pytest.mark.parametrize("kind", ["ones", "rank 3", "sparse", "hilbert"])
@pytest.mark.parametrize("tile,tiles", [(16, 8), (32, 3), (64, 3), (64, 8), (128, 3), (256, 2)])
def test_dependent_columns(avs_mod, tile, tiles, kind, dt, mode, tol):
    cuda()
    a = matrix(kind, tile * tiles).astype(dt)
    ref = sl.svdvals(a.astype(np.float64))
    got = avs_mod.my_CU_svdval(avs_mod.to_device(a), tile, precision=mode).cpu().numpy().astype(np.float64)
    assert np.max(np.abs(got - ref)) <= tol * ref[0]
    if mode is None:  # R^T R = A^T A, to the same bound
        f = avs_mod.to_device(a)
        avs_mod.tiled_QR(f, tile)
        r = np.triu(avs_mod.from_device(f)).astype(np.float64)
        a = a.astype(np.float64)
        assert np.max(np.abs(r.T @ r - a.T @ a)) <= 2 * tol * ref[0] ** 2


@pytest.mark.parametrize("mode", ["bf16x3", "tf32x3"])
@pytest.mark.parametrize("tile,tiles", [(128, 3), (256, 3)])
@pytest.mark.parametrize("kind", ["ones", "hilbert"])
def test_dependent_columns_tensor_core(avs_mod, kind, tile, tiles, mode):
    cuda()
    a = matrix(kind, tile * tiles).astype(np.float32)
    got = avs_mod.my_CU_svdval(avs_mod.to_device(a), tile, precision=mode).cpu().numpy().astype(np.float64)
    ref = sl.svdvals(a.astype(np.float64))
    assert np.max(np.abs(got - ref)) <= 1e-5 * ref[0]


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("tile,tiles", [(16, 8), (64, 5), (128, 3)])
def test_dependent_columns_other_forms(avs_mod, tile, tiles, dt):
    torch = cuda()
    n = tile * tiles
    a = np.asfortranarray(matrix("ones", n).astype(dt))
    d = avs_mod.to_device(a)
    single = avs_mod.my_CU_svdval(d, tile)
    other = avs_mod.to_device(np.random.default_rng(1).standard_normal((n, n)).astype(dt))
    outs = avs_mod.svdvals_batched([other, d, other, d], tiles=tile)
    assert torch.equal(outs[1], single) and torch.equal(outs[3], single)
    avs_mod.Blockbidiag(d, tile)
    h = a.copy(order="F")
    avs_mod.OOC_Bidiag(h, tile, device_bytes=6 * tile * n * h.itemsize + (1 << 20))
    assert np.array_equal(h, avs_mod.from_device(d))


@pytest.mark.parametrize("scale", [1e-18, 1e-19, 3e-20, 1e-20])
@pytest.mark.parametrize("tile,tiles", [(16, 3), (16, 8), (32, 3), (64, 3), (128, 3), (256, 2)])
def test_end_of_the_fp32_range(avs_mod, tile, tiles, scale):
    cuda()
    n = tile * tiles
    a = (np.random.default_rng(7).standard_normal((n, n)) * scale).astype(np.float32)
    f = avs_mod.to_device(a)
    try:
        avs_mod.Blockbidiag(f, tile)
    except avs_mod.AvsError as e:
        assert e.status == 4  # AVS_ERR_NONFINITE
        return
    band = np.triu(avs_mod.from_device(f)).astype(np.float64)
    band = (band - np.triu(band, tile + 1)) / scale
    a = a.astype(np.float64) / scale
    assert np.all(np.isfinite(band))
    assert np.max(np.abs(sl.svdvals(band) - sl.svdvals(a))) <= 1e-5 * sl.svdvals(a)[0]


@pytest.mark.parametrize("tile,tiles", [(16, 3), (16, 8), (32, 3), (64, 3), (128, 3)])
def test_end_of_the_fp32_range_in_double_float(avs_mod, tile, tiles):
    """Where FP32's range ends, double-float loses its second word: refused, not answered to
    a few digits (these Gaussian matrices have a column below 5e-20 in one of their panels)."""
    cuda()
    a = np.random.default_rng(7).standard_normal((tile * tiles, tile * tiles)) * 1e-19
    with pytest.raises(avs_mod.AvsError) as e:
        avs_mod.my_CU_svdval(avs_mod.to_device(a), tile, precision="fp64x2")
    assert e.value.status == 4  # AVS_ERR_NONFINITE
