"""Stage 3 at its edges: one to a few values, lane counts on both sides of their
limits, spectra with clusters, zeros and isolated tiny values, and bidiagonals
scaled near the ends of the exponent range, against LAPACK (relative to the
largest value: 1e-14, the bisection width of 2 eps plus the counts' rounding);
and a batch against its single calls."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu


def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def bidiagonal(n, kind):
    rng = np.random.default_rng(n)
    d, e = rng.standard_normal(n), rng.standard_normal(max(n - 1, 0))
    if kind == "cluster":
        d, e = np.ones(n), np.full(max(n - 1, 0), 1e-9)
    elif kind == "zeros":
        d[::3] = 0.0
        e[::5] = 0.0
    elif kind == "graded":
        d = 10.0 ** -np.linspace(0, 14, n)
        e = 0.5 * d[1:]
    return d, e


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -900, 2.0 ** 900])
@pytest.mark.parametrize("kind", ["gauss", "cluster", "zeros", "graded"])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 513, 1025])
def test_bidiagonal_values(avs_mod, n, kind, scale):
    torch = cuda()
    d, e = bidiagonal(n, kind)
    s = avs_mod.diag_lapack(torch.from_numpy(d * scale).cuda(), torch.from_numpy(e * scale).cuda()).cpu().numpy()
    ref = sl.svdvals(np.diag(d) + np.diag(e, 1))
    assert np.all(np.diff(s) <= 0)
    assert np.max(np.abs(s / scale - ref)) <= 1e-14 * ref[0]


def test_zero_bidiagonal(avs_mod):
    torch = cuda()
    z = torch.zeros(40, dtype=torch.float64, device="cuda")
    assert float(avs_mod.diag_lapack(z, z[:39]).abs().max()) == 0.0


@pytest.mark.parametrize("dt,tile,n,count", [(np.float32, 16, 48, 200), (np.float32, 64, 640, 24),
                                             (np.float64, 16, 64, 40)])
def test_batch_values_are_the_single_calls(avs_mod, dt, tile, n, count):
    torch = cuda()
    rng = np.random.default_rng(n)
    mats = [avs_mod.to_device(rng.standard_normal((n, n)).astype(dt)) for _ in range(count)]
    outs = avs_mod.svdvals_batched(list(mats), tiles=tile)
    for i in range(0, count, max(1, count // 12)):
        assert torch.equal(outs[i], avs_mod.my_CU_svdval(mats[i], tile))
