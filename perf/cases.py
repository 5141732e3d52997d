"""Performance cases of the tiled SVD: the calls a program makes through the
Python host mirror (``avs``), over the sizes, tiles, types and precision modes
it supports.

A case is a dict; ``kind`` says which entry point it calls:

* ``svd``    -- ``avs.my_CU_svdval`` on one matrix (device tensor, or a numpy
  host matrix with ``host``: the copies are then inside the call);
* ``batch``  -- ``avs.svdvals_batched`` on many matrices of mixed orders;
* ``serve``  -- ``avs.Server``: a burst of host requests of mixed orders and
  types, submitted and waited for;
* ``qr``     -- ``avs.tiled_QR`` (in place on a copy of the caller's matrix);
* ``bdsdc``  -- ``avs.diag_lapack``, the singular values of a bidiagonal.

Matrices are i.i.d. Gaussian N(0, 1/n) (``spectrum`` "gaussian") or
A = U diag(sigma) V^T with Haar U, V and sigma geometric from 1 to 1e-6
("geometric"), made on the GPU from the seed.
"""
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "avocado-sandwich_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import avs  # noqa: E402

_DTYPE = {"f32": torch.float32, "f64": torch.float64}
# Orders of the batched and served mixes, and the tiles a caller passes for
# them (a fixed rule: the autotuner times tiles, which is not part of a call).
_BATCH_TILE = {64: 32, 96: 16, 128: 32, 160: 32, 256: 32, 384: 64, 512: 64, 768: 64, 1024: 64}
_SERVER = None


def listed():
    return [
        # the smallest served request: latency of one small call, every launch counts
        {"name": "svd_f32_n128_t32", "kind": "svd", "dtype": "f32", "n": 128, "tile": 32, "precision": "default",
         "spectrum": "gaussian", "host": False},
        # ragged order (81 tiles of 16), the smallest tile the entry point takes
        {"name": "svd_f32_n1296_t16", "kind": "svd", "dtype": "f32", "n": 1296, "tile": 16, "precision": "default",
         "spectrum": "gaussian", "host": False},
        # the plain method: one 1024 x 1024 Float64 matrix, tile 64
        {"name": "svd_f64_n1024_t64", "kind": "svd", "dtype": "f64", "n": 1024, "tile": 64, "precision": "default",
         "spectrum": "gaussian", "host": False},
        # the Matrix{Float32} method: host matrix in, host values out
        {"name": "svd_f32_n2048_t64_host", "kind": "svd", "dtype": "f32", "n": 2048, "tile": 64,
         "precision": "default", "spectrum": "gaussian", "host": True},
        # FP32 with SIMT updates, prescribed spectrum, tile 128
        {"name": "svd_f32_n4096_t128_geo", "kind": "svd", "dtype": "f32", "n": 4096, "tile": 128,
         "precision": "default", "spectrum": "geometric", "host": False},
        # tensor-core updates at an odd number of tiles (45 x 128)
        {"name": "svd_bf16x3_n5760_t128", "kind": "svd", "dtype": "f32", "n": 5760, "tile": 128,
         "precision": "bf16x3", "spectrum": "gaussian", "host": False},
        # the headline: n = 16384, tile 256, split BF16
        {"name": "svd_bf16x3_n16384_t256", "kind": "svd", "dtype": "f32", "n": 16384, "tile": 256,
         "precision": "bf16x3", "spectrum": "gaussian", "host": False},
        # FP64-level accuracy on the FP32 pipe: how Float64 requests are served
        {"name": "svd_fp64x2_n2048_t128", "kind": "svd", "dtype": "f64", "n": 2048, "tile": 128,
         "precision": "fp64x2", "spectrum": "gaussian", "host": False},
        # random-matrix sampling: many small matrices of mixed orders in one call
        {"name": "batch_f32_192", "kind": "batch", "dtype": "f32", "count": 192, "orders": "64,128,256,512,1024"},
        # a burst of served requests, orders 128..1024, about 30% Float64
        {"name": "serve_32", "kind": "serve", "count": 32, "orders": "128,256,512,1024"},
        # tiled QR of a ragged order (15 x 128)
        {"name": "qr_f32_n1920_t128", "kind": "qr", "dtype": "f32", "n": 1920, "tile": 128, "precision": "default"},
        # the bidiagonal stage alone (LAPACK bdsdc's values)
        {"name": "bdsdc_n4096", "kind": "bdsdc", "n": 4096},
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _order(rng, tile, lo, hi):
    """A multiple of the tile (at least two tiles), log-uniform in [lo, hi]."""
    hi = max(hi // tile, 2)
    return tile * min(hi, max(2, round(_log_uniform(rng, max(lo, 2 * tile), hi * tile) / tile)))


def draw(rng):
    kind = rng.choice(["svd"] * 7 + ["batch", "serve", "qr", "qr", "bdsdc"])
    if kind == "svd":
        mode = rng.choice(["default", "default", "default", "f64", "fp64x2", "tf32x3", "bf16x3", "bf16x3"])
        if mode == "f64":
            tile, dtype, precision = rng.choice([16, 32, 64, 128]), "f64", "default"
            n = _order(rng, tile, 64, 1600)
        elif mode == "fp64x2":
            tile, dtype, precision = rng.choice([32, 64, 128]), "f64", mode
            n = _order(rng, tile, 128, 3072)
        elif mode == "default":
            tile, dtype, precision = rng.choice([16, 32, 64, 128, 256]), "f32", mode
            n = _order(rng, tile, 64, {16: 2048, 32: 4096}.get(tile, 6144))
        else:
            tile, dtype, precision = rng.choice([128, 256]), "f32", mode
            n = _order(rng, tile, 1024, 12288)
        return {"kind": "svd", "dtype": dtype, "n": n, "tile": tile, "precision": precision,
                "spectrum": rng.choice(["gaussian", "gaussian", "geometric"]), "host": rng.random() < 0.25}
    if kind == "batch":
        orders = sorted(rng.sample(sorted(_BATCH_TILE), rng.randint(1, 5)))
        count = int(round(_log_uniform(rng, 16, 256)))
        return {"kind": "batch", "dtype": rng.choice(["f32", "f32", "f64"]) if max(orders) <= 256 else "f32",
                "count": count, "orders": ",".join(map(str, orders))}
    if kind == "serve":
        return {"kind": "serve", "count": rng.randint(8, 56),
                "orders": ",".join(map(str, sorted(rng.sample([128, 256, 512, 1024], rng.randint(2, 4)))))}
    if kind == "qr":
        dtype = rng.choice(["f32", "f32", "f64"])
        tile = rng.choice([16, 32, 64, 128, 256])
        n = _order(rng, tile, 96, {16: 1024, 32: 1536}.get(tile, 2048) if dtype == "f32" else 1024)
        return {"kind": "qr", "dtype": dtype, "n": n, "tile": tile, "precision": "default"}
    return {"kind": "bdsdc", "n": int(round(_log_uniform(rng, 50, 6000)))}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _haar(n, gen):
    # QR in FP32 above n = 2048: the factors need to be random, not exact (the
    # input is whatever the product rounds to), and FP64 QR is slow there
    q, r = torch.linalg.qr(torch.randn((n, n), generator=gen, device="cuda",
                                       dtype=torch.float64 if n <= 2048 else torch.float32))
    return q * torch.sign(torch.diagonal(r))[None, :]


def _matrix(case, seed):
    n, gen = case["n"], _gen(seed)
    dt = _DTYPE[case["dtype"]]
    if case["spectrum"] == "geometric":
        u, v = _haar(n, gen), _haar(n, gen)
        s = 1e-6 ** (torch.arange(n, device="cuda", dtype=u.dtype) / (n - 1.0))
        return ((v * s[None, :]) @ u.T).to(dt).contiguous()
    return torch.randn((n, n), generator=gen, device="cuda", dtype=dt) / n ** 0.5


def _orders(case):
    return [int(x) for x in case["orders"].split(",")]


def _batch(case, seed):
    """The orders in turn through the batch, so that every seed is the same amount of work."""
    gen, dt = _gen(seed), _DTYPE[case["dtype"]]
    orders = _orders(case)
    ns = [orders[i % len(orders)] for i in range(case["count"])]
    return ns, [torch.randn((n, n), generator=gen, device="cuda", dtype=dt) / n ** 0.5 for n in ns]


def _requests(case, seed):
    orders = _orders(case)
    rng = np.random.default_rng(int(seed))
    reqs = []
    for i in range(case["count"]):
        n = orders[(i * 7) % len(orders)]
        dt = np.float64 if i % 10 in (1, 4, 8) else np.float32
        reqs.append(np.asfortranarray((rng.standard_normal((n, n)) / n ** 0.5).astype(dt)))
    return reqs


def _bidiagonal(case, seed):
    """d, e of the Golub-Kahan bidiagonal of an n x n Gaussian matrix N(0, 1/n):
    independent chi variables (what stage 2 hands to the last stage)."""
    n = case["n"]
    rng = np.random.default_rng(int(seed))
    d = np.sqrt(rng.chisquare(np.arange(n, 0, -1.0)) / n)
    e = np.sqrt(rng.chisquare(np.arange(n - 1, 0, -1.0)) / n)
    return torch.from_numpy(d).cuda(), torch.from_numpy(e).cuda()


def _server():
    global _SERVER
    if _SERVER is None:  # a program keeps one server
        _SERVER = avs.Server(workers=4)
    return _SERVER


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "svd":
        a = _matrix(case, seed)  # the matrix column-major: a is its transpose
        st["a"] = a.cpu().numpy().T if case["host"] else a
    elif kind == "batch":
        st["orders"], st["mats"] = _batch(case, seed)
        st["tiles"] = [_BATCH_TILE[n] for n in st["orders"]]
    elif kind == "serve":
        st["reqs"], st["server"] = _requests(case, seed), _server()
    elif kind == "qr":
        st["a"] = torch.randn((case["n"], case["n"]), generator=_gen(seed), device="cuda", dtype=_DTYPE[case["dtype"]])
    else:
        st["d"], st["e"] = _bidiagonal(case, seed)
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "svd":
        return avs.my_CU_svdval(state["a"], case["tile"], precision=case["precision"])
    if kind == "batch":
        outs = avs.svdvals_batched(list(state["mats"]), tiles=state["tiles"])
        return torch.cat(outs)
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(a) for a in state["reqs"]]
        return [srv.wait(i)[0] for i in ids]
    if kind == "qr":
        a = state["a"].clone()
        tau = avs.tiled_QR(a, case["tile"], precision=case["precision"])
        return {"factors": a, "tau": tau}
    return avs.diag_lapack(state["d"], state["e"])


def work(case):
    """Bytes: inputs read once, outputs written once.  Flops: the textbook count
    of the path ((8/3) n^3 for the reduction of an SVD, (4/3) n^3 for QR; for
    the values of a bidiagonal about 50 Sturm counts of 2n pivots each)."""
    kind = case["kind"]
    if kind == "svd":
        n, w = case["n"], 4 if case["dtype"] == "f32" else 8
        return {"bytes": w * (n * n + n), "flops": 8.0 / 3.0 * n ** 3}
    if kind in ("batch", "serve"):
        orders = _orders(case)
        by = fl = 0.0
        for i in range(case["count"]):
            if kind == "batch":
                n, w = orders[i % len(orders)], 4 if case["dtype"] == "f32" else 8
            else:
                n, w = orders[(i * 7) % len(orders)], 8 if i % 10 in (1, 4, 8) else 4
            by += w * (n * n + n)
            fl += 8.0 / 3.0 * n ** 3
        return {"bytes": by, "flops": fl}
    if kind == "qr":
        n, w = case["n"], 4 if case["dtype"] == "f32" else 8
        return {"bytes": 2 * w * n * n + w * n * (n // case["tile"]), "flops": 4.0 / 3.0 * n ** 3}
    n = case["n"]
    return {"bytes": 8 * (3 * n - 1), "flops": 50.0 * 2 * n * 3 * n}


def _svals(a):
    """Singular values in FP64 (LAPACK / cuSOLVER through torch)."""
    a = a.to(torch.float64)
    if a.shape[-1] <= 1536:
        return torch.linalg.svdvals(a.cpu())
    return torch.linalg.svdvals(a.cuda(), driver="gesvd")


def _exact_qr(a, tile):
    """The flat-tree tiled QR in FP64: LAPACK's geqrf on the diagonal tile, then
    on [R; tile] down the panel (same reflector normalisation as LAPACK)."""
    n, b = a.shape[0], tile
    nt = n // b
    tau = torch.zeros(nt, nt, b, dtype=torch.float64)

    def factor(rows, c0, k, r):
        x = torch.cat([a[q:q + b] for q in rows])
        p = x[:, c0:c0 + b].clone()
        if len(rows) == 2:
            p[:b] = torch.triu(p[:b])
        f, t = torch.geqrf(p)
        tau[k, r] = t
        if c0 + b < n:
            x[:, c0 + b:] = torch.ormqr(f, t, x[:, c0 + b:].contiguous(), left=True, transpose=True)
        top = torch.triu(f[:b]) + torch.tril(x[:b, c0:c0 + b], -1) if len(rows) == 2 else f[:b]
        x[:b, c0:c0 + b] = top
        if len(rows) == 2:
            x[b:, c0:c0 + b] = f[b:]
        for i, q in enumerate(rows):
            a[q:q + b] = x[i * b:(i + 1) * b]

    for k in range(nt):
        factor([k * b], k * b, k, k)
        for r in range(k + 1, nt):
            factor([k * b, r * b], k * b, k, r)
    return a, tau.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "svd":
        if case["n"] > 6144:
            return None
        return _svals(_matrix(case, seed))
    if kind == "batch":
        return torch.cat([_svals(m) for m in _batch(case, seed)[1]])
    if kind == "serve":
        return [_svals(torch.from_numpy(np.ascontiguousarray(a))) for a in _requests(case, seed)]
    if kind == "qr":
        a = torch.randn((case["n"], case["n"]), generator=_gen(seed), device="cuda", dtype=_DTYPE[case["dtype"]])
        f, tau = _exact_qr(a.cpu().to(torch.float64).T.contiguous(), case["tile"])
        return {"factors": f.T.contiguous(), "tau": tau}
    d, e = (x.cpu() for x in _bidiagonal(case, seed))
    return torch.linalg.svdvals(torch.diag(d) + torch.diag(e, 1)) if case["n"] <= 1536 else \
        torch.linalg.svdvals((torch.diag(d) + torch.diag(e, 1)).cuda(), driver="gesvd")
