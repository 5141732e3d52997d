"""The captured graphs of a batched call belong to a bisection width: a call with
another width on the same handle gets its own values, not those of the width that
was captured first (each batch = its single calls with that width, bit for bit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_batched_calls_of_other_widths(avs_mod, dt):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    h = avs_mod.Handle()
    try:
        rng = np.random.default_rng(9)
        mats = [avs_mod.to_device(rng.standard_normal((96, 96)).astype(dt)) for _ in range(3)]
        for rel_tol in (1e-3, 0.0, 1e-7, 1e-3):
            outs = avs_mod.svdvals_batched(list(mats), tiles=16, handle=h, rel_tol=rel_tol)
            for a, s in zip(mats, outs):
                assert torch.equal(s, avs_mod.my_CU_svdval(a, 16, handle=h, rel_tol=rel_tol))
    finally:
        h.close()
