"""The bidiagonal entry point at the limits of its input: infinite and NaN entries,
entries whose Gershgorin bound overflows, bounds next to the largest double.
Expected: an infinite entry gives infinite values; finite entries give their values
(LAPACK's of the matrix scaled by a power of two, 1e-14 of the largest); a NaN entry
gives what the allocation-free entry point gives, within the default width of both.
And at widths below the default: ``rel_tol`` is the width of the final bracket relative
to the bound whatever it is, so small values keep their relative accuracy.  The counts
are exact for off-diagonals within 2^-46, i.e. a value moves by 2n 2^-46 of itself at
most.  The Gershgorin bound is at most twice the largest value here."""
import ctypes

import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")


def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def values(avs_mod, d, e, rel_tol=0.0):
    torch = cuda()
    d, e = (torch.tensor(x, dtype=torch.float64, device="cuda") for x in (d, e))
    return avs_mod.diag_lapack(d, e, rel_tol).cpu().numpy()


def values_noalloc(avs_mod, d, e, rel_tol=0.0):
    torch = cuda()
    d, e = (torch.tensor(x, dtype=torch.float64, device="cuda") for x in (d, e))
    s = torch.empty_like(d)
    torch.cuda.synchronize()
    rc = avs_mod.lib().avs_bidiag_svals_noalloc(d.numel(), ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(e.data_ptr()),
                                                ctypes.c_void_p(s.data_ptr()), rel_tol, None)
    assert rc == 0
    return s.cpu().numpy()


@pytest.mark.parametrize("d,e", [((3.0, INF, 2.0, 0.5), (0.1, 0.2, 0.3)), ((3.0, 1.0, 2.0, 0.5), (0.1, -INF, 0.3)),
                                 ((NAN, INF, 2.0), (0.1, 0.2)), ((INF,), ())])
def test_infinite_entries(avs_mod, d, e):
    assert np.all(values(avs_mod, d, e) == INF)
    assert np.all(values_noalloc(avs_mod, d, e) == INF)


@pytest.mark.parametrize("d,e", [((3.0, NAN, 2.0, 0.5), (0.1, 0.2, 0.3)), ((3.0, 1.0, 2.0, 0.5), (0.1, NAN, 0.3)),
                                 ((NAN, 1.0, 2.0, 0.5), (0.1, 0.2, 0.3)), ((NAN,), ())])
def test_nan_entries(avs_mod, d, e):
    got, ref = values(avs_mod, d, e), values_noalloc(avs_mod, d, e)
    assert np.max(np.abs(got - ref)) <= 1e-14 * np.max(ref)


@pytest.mark.parametrize("d,e", [((1e308, 1e308), (1e308,)), ((-1e308, 0.7e308, 1e300), (0.9e308, 0.0)),
                                 ((1.79e308,), ()), ((np.finfo(np.float64).max, 1.0), (0.0,)),
                                 ((np.finfo(np.float64).max * (1 - 1e-7), 1e308), (0.0,))])
def test_bounds_that_overflow(avs_mod, d, e):
    s = 2.0 ** -1000
    ref = sl.svdvals(np.diag(np.array(d) * s) + np.diag(np.array(e) * s, 1))
    got = values(avs_mod, d, e) * s
    assert np.max(np.abs(got - ref)) <= 1e-14 * ref[0]


@pytest.mark.parametrize("rel_tol", [1e-17, 1e-20, 1e-30])
def test_width_below_the_grid_diagonal(avs_mod, rel_tol):
    d = 10.0 ** -np.arange(0, 33, 2.0)
    got = values(avs_mod, d, np.zeros(d.size - 1), rel_tol)
    assert np.all(np.abs(got - d) <= rel_tol * d[0] + 2 * d.size * 2.0 ** -46 * d)


@pytest.mark.parametrize("rel_tol", [1e-18, 1e-30])
@pytest.mark.parametrize("n", [4, 50, 600])
def test_width_below_the_grid_graded(avs_mod, n, rel_tol):
    d = 10.0 ** -np.linspace(0, 28, n)
    e = 0.5 * d[1:]
    got, ref = values(avs_mod, d, e, rel_tol), values_noalloc(avs_mod, d, e, rel_tol)
    assert np.all(np.diff(got) <= 0)
    assert np.all(np.abs(got - ref) <= 2 * rel_tol * 2 * d[0] + 4 * n * 2.0 ** -46 * ref)


def test_width_below_the_grid_zero_value(avs_mod):
    got = values(avs_mod, (2.0, 1.0, 0.0, 1.0), (1.0, 1.0, 1.0), 1e-30)
    assert got[3] <= 1e-30 * 4.0


@pytest.mark.parametrize("batch", [False, True])
def test_width_below_the_grid_whole_call(avs_mod, batch):
    torch = cuda()
    d = 10.0 ** -np.linspace(0, 20, 64)
    a = torch.diag(torch.from_numpy(d)).cuda()
    if batch:
        got = avs_mod.svdvals_batched([a, a.clone()], tiles=16, rel_tol=1e-26)[1]
    else:
        got = avs_mod.my_CU_svdval(a, 16, rel_tol=1e-26)
    assert np.all(np.abs(got.cpu().numpy() - d) <= 1e-26 + 2 * d.size * 2.0 ** -46 * d)


def test_narrowest_width_in_double_float(avs_mod):
    """A width of 1e-15 of the bound (here 0.9): the values, midpoints of brackets no wider
    than that, cannot all be midpoints of cells of 2^-47."""
    torch = cuda()
    d = np.random.default_rng(5).uniform(0.0, 0.9, 64)
    d[0] = 0.9
    a = torch.diag(torch.from_numpy(d)).cuda()
    got = avs_mod.my_CU_svdval(a, 16, precision="fp64x2", rel_tol=1e-15).cpu().numpy()
    assert np.any((got * 2.0 ** 48) % 1.0 != 0.0)
    assert np.max(np.abs(got - np.sort(d)[::-1])) <= 2e-14
