"""Forms that the kernels' other tests leave out, each bit for bit against the call by
itself: calls of other tiles, types and precisions on one handle in between (the
buffers that the stages share, and the panel's tagged words, on the second stream of
the tensor-core path too); batches of Float64 matrices in double-float, tiles 64 and
128, whose block stage runs over the whole batch; and batches on both sides of the
count from which the FP32 updates of tiles 32 and 64 give a CTA all tiles of a strip
(304 strips, i.e. matrices times strips of 64 columns)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


CALLS = [(np.float32, None, 16, 7), (np.float64, None, 64, 3), (np.float32, "bf16x3", 128, 5), (np.float64, "fp64x2", 32, 5),
         (np.float32, "tf32x3", 256, 3), (np.float64, "fp64x2", 128, 3), (np.float32, None, 64, 5), (np.float64, None, 16, 9),
         (np.float64, "fp64x2", 256, 2), (np.float32, None, 256, 2), (np.float32, "bf16x3", 256, 2)]


def test_calls_of_other_kinds_in_between(avs_mod):
    torch = cuda()
    h = avs_mod.Handle()
    try:
        rng = np.random.default_rng(3)
        mats = [avs_mod.to_device(rng.standard_normal((t * k, t * k)).astype(dt)) for dt, _, t, k in CALLS]

        def run(i):
            dt, prec, tile, _ = CALLS[i]
            f = mats[i].clone()
            tau = avs_mod.tiled_QR(f, tile, precision=prec, handle=h)
            return avs_mod.my_CU_svdval(mats[i], tile, precision=prec, handle=h), f, tau

        first = [run(i) for i in range(len(CALLS))]
        for i in list(rng.permutation(len(CALLS))) + list(range(len(CALLS)))[::-1]:
            assert all(torch.equal(a, b) for a, b in zip(run(i), first[i])), CALLS[i]
    finally:
        h.close()


@pytest.mark.parametrize("tile,n,count", [(64, 192, 5), (64, 640, 3), (128, 256, 4), (128, 640, 3), (256, 512, 2)])
def test_double_float_batches(avs_mod, tile, n, count):
    torch = cuda()
    rng = np.random.default_rng(n + tile)
    mats = [avs_mod.to_device(rng.standard_normal((n, n))) for _ in range(count)]
    outs = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(count)]
    h = avs_mod.default_handle()
    ptrs = lambda ts: (ctypes.c_void_p * count)(*[t.data_ptr() for t in ts])
    o = avs_mod.Opts(avs_mod._prec("fp64x2"), 0, 0.0,
                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    r = avs_mod.Report()
    rc = avs_mod.lib().avs_svdvals_batched_dev_d(h.ptr, count, (ctypes.c_int64 * count)(*[n] * count),
                                                 (ctypes.c_int64 * count)(*[n] * count),
                                                 (ctypes.c_int32 * count)(*[tile] * count), ptrs(mats), ptrs(outs),
                                                 ctypes.byref(o), ctypes.byref(r))
    assert rc == 0
    for a, s in zip(mats, outs):
        assert torch.equal(s, avs_mod.my_CU_svdval(a, tile, precision="fp64x2"))


@pytest.mark.parametrize("tile,n,count", [(32, 160, 160), (32, 320, 64), (64, 448, 64), (64, 704, 33)])
def test_update_all_tiles_in_a_cta(avs_mod, tile, n, count):
    torch = cuda()
    assert ((n - tile + 63) // 64) * count >= 304
    rng = np.random.default_rng(n)
    mats = [avs_mod.to_device(rng.standard_normal((n, n)).astype(np.float32)) for _ in range(4)]
    outs = avs_mod.svdvals_batched([mats[i % 4] for i in range(count)], tiles=tile)
    for i in range(4):
        single = avs_mod.my_CU_svdval(mats[i], tile)
        assert all(torch.equal(outs[q], single) for q in range(i, count, 4))
