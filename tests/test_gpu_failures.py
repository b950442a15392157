"""Failure handling without a GPU fault: an allocation failure injected on the host side of the
context (TT_ERR_NOMEM, the context stays usable), and a bounded device wait that runs out
(TT_ERR_TIMEOUT read from the status word, the context stays usable)."""
import time

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _ttr():
    import tensor_train_ring_decompositions_hpc_gpu_b200 as ttr
    return ttr


def _small_tensor(gpu, seed=3):
    import torch
    x = oracle.make_tt_tensor([16, 16, 16, 16], [1, 4, 4, 4, 1], 1e-4, seed=seed)
    return torch.from_numpy(np.asfortranarray(x, dtype=np.float32)).to(gpu), x


def test_injected_allocation_failure(gpu):
    ttr = _ttr()
    from tensor_train_ring_decompositions_hpc_gpu_b200 import _lib
    lib = ttr.lib()
    # a fresh context on another stream, so the shared context's workspace is not already large
    import torch
    import ctypes as C
    stream = torch.cuda.Stream(gpu)
    ctx = C.c_void_p()
    assert lib.tt_ctx_create(C.byref(ctx), gpu.index or 0, C.c_void_p(stream.cuda_stream)) == 0
    try:
        xd, x = _small_tensor(gpu)
        n, r = [16] * 4, [1, 4, 4, 4, 1]
        cores = [torch.empty(r[k] * n[k] * r[k + 1], device=gpu) for k in range(4)]
        ptrs = (C.c_void_p * 4)(*[t.data_ptr() for t in cores])
        o = ttr._opts("auto", "edrsvd", 8, 0, 1, 0, 40)
        assert lib.tt_ctx_set_alloc_limit(ctx, 4096) == 0
        rc = lib.tt_svd(ctx, C.c_void_p(xd.data_ptr()), 4, _lib.int_array(n), _lib.int_array(r), C.byref(o), ptrs,
                        None)
        assert rc == 5 and b"allocation limit" in lib.tt_last_error()  # TT_ERR_NOMEM
        assert lib.tt_ctx_set_alloc_limit(ctx, 0) == 0
        rc = lib.tt_svd(ctx, C.c_void_p(xd.data_ptr()), 4, _lib.int_array(n), _lib.int_array(r), C.byref(o), ptrs,
                        None)
        assert rc == 0, lib.tt_last_error()
        torch.cuda.synchronize(gpu)
        g = [ttr._core_view(cores[k], r[k], n[k], r[k + 1]).double().cpu().numpy() for k in range(4)]
        assert oracle.rel_error(x, oracle.tt_full(g)) < 1e-3
    finally:
        lib.tt_ctx_destroy(ctx)


def test_wait_limit_runs_out_and_context_survives(gpu):
    ttr = _ttr()
    lib = ttr.lib()
    ctx = ttr._ctx_for(gpu.index or 0)
    assert lib.tt_ctx_set_wait_limit(ctx, 5_000_000) == 0  # 5 ms
    try:
        t0 = time.time()
        rc = lib.tt_k_wait_selftest(ctx)
        dt = time.time() - t0
        assert rc == 7 and b"device status 7" in lib.tt_last_error()  # TT_ERR_TIMEOUT
        assert dt < 1.0
    finally:
        assert lib.tt_ctx_set_wait_limit(ctx, 0) == 0
    # the context and the device stay usable
    xd, x = _small_tensor(gpu, seed=5)
    res = ttr.tt_svd(xd, [1, 4, 4, 4, 1])
    g = [c.double().cpu().numpy() for c in res.cores]
    assert oracle.rel_error(x, oracle.tt_full(g)) < 1e-3


@pytest.mark.parametrize("shape,rank,bounds,gemm", [
    ((17, 8, 75776), 16, (17, 24), "fp32"),   # 128 rows instead of 136: more splits of the sketch
    ((33, 32, 20000), 32, (33, 24), "tc"),    # 1024 rows instead of 1056, the same on the tensor cores
    ((17, 8, 200), 12, (17, 40), "fp32"),     # 96 rows instead of 136: an exact step and its eigen-solve
])
def test_tolerance_run_whose_ranks_shrink(gpu, monkeypatch, shape, rank, bounds, gemm):
    """The first rank comes out below its bound, and the step after it needs more scratch than it was planned with: a
    fresh context has it."""
    import torch
    ttr = _ttr()
    monkeypatch.setattr(ttr, "_CTX", {})
    g = torch.Generator(device=gpu).manual_seed(sum(shape))
    a = torch.randn(shape[0], rank, generator=g, device=gpu)
    b = torch.randn(rank * shape[1], 12, generator=g, device=gpu)
    c = torch.randn(12, shape[2], generator=g, device=gpu)
    x = torch.einsum("ir,rjs,sk->ijk", a, b.view(rank, shape[1], 12), c)
    res = ttr.tt_svd(x, [1, *bounds, 1], eps=1e-3, gemm=gemm)
    assert res.ranks == [1, rank, 12, 1]
    assert ttr.rel_error(x, res.cores) < 1e-3


def test_tolerance_run_at_its_allocation_limit(gpu, monkeypatch):
    """The same where nothing may be allocated beyond what the plan takes: the sketch makes do with fewer splits."""
    import torch
    ttr = _ttr()
    g = torch.Generator(device=gpu).manual_seed(4)
    a = torch.randn(17, 16, generator=g, device=gpu)
    b = torch.randn(16 * 8, 12, generator=g, device=gpu)
    c = torch.randn(12, 75776, generator=g, device=gpu)
    x = torch.einsum("ir,rjs,sk->ijk", a, b.view(16, 8, 12), c)
    low, high = 1 << 20, 1 << 30
    while high - low > 1 << 20:  # the least limit, to 1 MiB, that a run which keeps its ranks needs
        mid = (low + high) // 2
        monkeypatch.setattr(ttr, "_CTX", {})
        assert ttr.lib().tt_ctx_set_alloc_limit(ttr._ctx_for(0), mid) == 0
        try:
            ttr.tt_svd(x, [1, 17, 24, 1], eps=1e-9)
            high = mid
        except ttr._lib.TTError:
            low = mid
    monkeypatch.setattr(ttr, "_CTX", {})
    assert ttr.lib().tt_ctx_set_alloc_limit(ttr._ctx_for(0), high) == 0
    res = ttr.tt_svd(x, [1, 17, 24, 1], eps=1e-3, gemm="fp32")
    assert res.ranks == [1, 16, 12, 1]


@pytest.mark.parametrize("call", ["tt", "tr", "eps", "sketch", "project"])
def test_fewer_splits_under_an_allocation_limit(gpu, monkeypatch, call):
    """Sketches and projections split their long side for speed.  Limits between the scratch of all these splits and
    that of fewer: the call runs, and to the same result."""
    import torch
    ttr = _ttr()
    g = torch.Generator(device=gpu).manual_seed(3)
    def rand(*shape):
        return torch.randn(*shape, generator=g, device=gpu)
    if call in ("sketch", "project"):
        m, n, N, limit = (50, 9469, 111, 7_650_000) if call == "sketch" else (225, 21602, 53, 2_100_000)
        a, w = rand(n, m).t(), rand(N, n if call == "sketch" else m).t()
        def run():
            return [getattr(ttr, call)(a, w, "fp32")]
    else:
        n, limit = {"tt": ((137, 110, 312), 20_100_000), "tr": ((140, 153, 251), 13_700_000),
                    "eps": ((144, 303, 132), 18_050_000)}[call]
        x = torch.einsum("ir,rjs,sk->kji", rand(n[0], 5), rand(5, n[1], 5), rand(5, n[2])).permute(2, 1, 0)
        x = x + 1e-4 * rand(n[2], n[1], n[0]).permute(2, 1, 0)
        def run():
            if call == "tr":
                res = ttr.tr_svd(x, [1, 1, 1, 1], gemm="fp32", power_iters=1, oversample=20)
            elif call == "tt":
                res = ttr.tt_svd(x, [1, 17, 17, 1], gemm="fp32", power_iters=1)
            else:
                res = ttr.tt_svd(x, [1, 5, 5, 1], eps=1e-2, oversample=20)
            return [torch.as_tensor(np.asarray(s)[:r]) for s, r in zip(res.sigmas, res.ranks[1:])]
    monkeypatch.setattr(ttr, "_CTX", {})
    want = run()
    monkeypatch.setattr(ttr, "_CTX", {})
    assert ttr.lib().tt_ctx_set_alloc_limit(ttr._ctx_for(0), limit) == 0
    for u, v in zip(want, run()):  # FP32 sums in another order
        assert float((u - v).abs().max()) <= 1e-5 * float(u.abs().max())
