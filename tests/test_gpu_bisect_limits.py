"""The bidiagonal entry point at the limits of its input: infinite and NaN entries,
entries whose Gershgorin bound overflows, bounds next to the largest double.
Expected: an infinite entry gives infinite values; finite entries give their values
(LAPACK's of the matrix scaled by a power of two, 1e-14 of the largest); a NaN entry
gives what the allocation-free entry point gives, within the default width of both."""
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
