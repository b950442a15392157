"""Precision that the decompositions hold: bounds from the rounding of the stored results, against NumPy in FP64."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

U32 = 2.0 ** -24  # unit roundoff of FP32


def _ttr():
    import tensor_train_ring_decompositions_hpc_gpu_b200 as ttr
    return ttr


def _dev(x, dev, dtype=np.float32):
    import torch
    return torch.from_numpy(np.asfortranarray(x, dtype=dtype)).to(dev)


@pytest.mark.parametrize("shape,ranks", [
    ((24, 24, 24, 24), (1, 24, 24, 24, 1)),   # 576 rows, 32 columns: one CholeskyQR launch
    ((256, 64, 48), (1, 16, 20, 1)),          # 24 columns of 256 and of 1024 rows
    ((110, 100, 20, 60), (1, 62, 66, 30, 1)),  # 6200 rows, 74 columns: more than one launch holds
    ((600, 96, 20), (1, 88, 18, 1)),          # 96 columns of 600 rows: rows multiplied by an inverse
])
@pytest.mark.parametrize("power", [0, 1])
def test_fp32_bases_are_orthonormal(gpu, shape, ranks, power):
    """Plain FP32 and fixed ranks.  A basis of m rows whose entries carry independent roundings (its own, those of
    Q and of E: 3 u at most together) has U^T U = I to 2 x 3 u |u_i o u_j| ~ 6 u sqrt(3 / m); 2x that is allowed.  A
    column of Q that is off in length by half an ulp in every row is off by u whatever m is."""
    x = oracle.make_tt_tensor(list(shape), list(ranks), 1e-4, seed=sum(shape))
    res = _ttr().tt_svd(_dev(x, gpu), list(ranks), gemm="fp32", oversample=8, power_iters=power)
    for k, c in enumerate(res.cores[:-1]):
        u = c.double().cpu().numpy().reshape(-1, c.shape[2], order="F")
        if u.shape[0] > 4 * u.shape[1] and u.shape[0] > 130:  # sketched steps
            defect = np.abs(u.T @ u - np.eye(u.shape[1])).max()
            assert defect <= 12 * U32 * np.sqrt(3.0 / u.shape[0]), (k, u.shape, defect)


def _fill_shared_memory_with_nan(dev):
    """Grams of NaN in either layout: what a later kernel finds in shared memory that it does not write is NaN."""
    import ctypes as C
    import torch
    ttr = _ttr()
    z = torch.full((200000, 128), float("nan"), device=dev)
    w = torch.empty((128, 128), dtype=torch.float64, device=dev)
    for rs, cs in ((128, 1), (1, 200000)):
        ttr._lib.check(ttr.lib().tt_k_gram_tall(ttr._ctx_for(0), C.c_void_p(z.data_ptr()), 200000, 128, rs, cs,
                                                C.c_void_p(w.data_ptr())))


@pytest.mark.parametrize("n,N", [(200000, 3), (100000, 7), (60000, 10), (60000, 27), (60001, 54), (60000, 101)])
def test_cholqr2_tall_ragged(gpu, n, N):
    """More rows than one launch holds and widths that are no multiple of 8, after a kernel that left NaN in shared
    memory.  Bounds as in test_cholqr2_edges."""
    import torch
    g = torch.Generator(device="cpu").manual_seed(n + N)
    y = torch.randn((N, n), generator=g).to(gpu).t()
    yd = y.double()
    _fill_shared_memory_with_nan(gpu)
    q, r = _ttr().cholqr2(y)
    qd = q.double()
    tol = 4 * U32 * N * max(1.0, np.sqrt(N))
    eye = torch.eye(N, dtype=torch.float64, device=gpu)
    assert float(torch.linalg.norm(qd.t() @ qd - eye)) <= tol
    assert float(torch.linalg.norm(qd @ r - yd)) <= tol * float(torch.linalg.norm(yd))


@pytest.mark.parametrize("n,N", [(8192, 1), (8193, 1), (8192, 12), (8193, 12), (16411, 2), (12001, 40)])
def test_cholqr2_around_the_rows_of_one_launch(gpu, n, N):
    """Both sides of the row count above which several launches are taken although one would hold the rows."""
    test_cholqr2_tall_ragged(gpu, n, N)


@pytest.mark.parametrize("n,N", [(256, 65), (400, 72), (300, 77), (462, 80)])
def test_cholqr2_wide_rows_are_solved(gpu, n, N):
    """65 to 80 columns of few rows: q R = y is solved row by row, like the narrower ones, and not multiplied by an
    inverse rounded to FP32.  R = 1 / 2 x normal above a unit diagonal has a condition of 1e4 and more.  Solving leaves
    Q (Q^T Y) - Y at the rounding of two passes' sums of N / 4 terms, 2 u sqrt(N / 4) of |Y|, of which 2x is allowed; a
    rounded inverse leaves u |Y R^-1| |R|, several times that bound."""
    import ctypes as C
    import torch
    ttr = _ttr()
    rng = np.random.default_rng(N)
    r = np.triu(rng.standard_normal((N, N)), 1) * 0.5 + np.diag(np.ones(N))
    q0 = np.linalg.qr(rng.standard_normal((n, N)))[0]
    y = (q0 @ r).astype(np.float32)
    yt = torch.from_numpy(np.ascontiguousarray(y.T)).to(gpu)
    ttr._lib.check(ttr.lib().tt_k_cholqr2(ttr._ctx_for(0), C.c_void_p(yt.data_ptr()), n, N, n, None))
    q = yt.t().double().cpu().numpy()
    yd = y.astype(np.float64)
    assert np.linalg.norm(q @ (q.T @ yd) - yd) <= 4 * U32 * np.sqrt(N / 4) * np.linalg.norm(yd)


@pytest.mark.parametrize("m", [17, 30, 31])
def test_adaptive_gram_of_unaligned_rows(gpu, m):
    """A tolerance run reads the discarded energy off the Gram of its first unfolding: 1e-8 of the whole here, of rows
    that are almost constant, so that FP32 products and sums would all round the same way (1e-7).  FP64 ones leave
    2^-53 of the whole per term, n m^2 terms at the worst: 1e-4 of the discarded energy at most."""
    n = 70000
    rng = np.random.default_rng(m)
    x = ((1.1 + 0.01 * np.arange(m))[:, None] * 0.9 * np.ones(n) + 1e-4 * rng.standard_normal((m, n))).astype(np.float32)
    res = _ttr().tt_svd(_dev(x, gpu), [1, 1, 1], eps=1e-3)
    lam = np.linalg.eigvalsh(x.astype(np.float64) @ x.T.astype(np.float64))
    want = np.sqrt(lam[:-1].sum() / lam.sum())
    assert abs(res.est_rel_err - want) <= 1e-4 * want


@pytest.mark.parametrize("shape,rank", [((9, 5, 9, 4), 2), ((7, 11, 5), 3), ((18, 10, 23, 6), 5), ((30, 7, 31), 6)])
def test_grams_of_odd_rows_do_not_overflow(gpu, shape, rank):
    """Rows that are no multiple of 4: values of about 2^62, sixteen of whose squares add up beyond FP32.  Scaling by a
    power of two changes no rounding, so the singular values are those of the tensor as it is, times that."""
    import torch
    ranks = [1] + [rank] * (len(shape) - 1) + [1]
    x = _dev(oracle.make_tt_tensor(list(shape), ranks, 1e-2, seed=sum(shape)), gpu)
    x = 1.0 + 0.25 * x / x.abs().max()
    one = _ttr().tt_svd(x, ranks, gemm="fp32")
    big = _ttr().tt_svd(x * 2.0 ** 62, ranks, gemm="fp32")
    for k, (a, b) in enumerate(zip(one.sigmas, big.sigmas)):
        a, b = np.asarray(a)[:ranks[k + 1]], np.asarray(b)[:ranks[k + 1]] / 2.0 ** 62
        assert np.abs(a - b).max() <= 1e-6 * a.max(), (k, a, b)
    assert all(torch.isfinite(c).all() for c in big.cores)


@pytest.mark.parametrize("m,n2,n3", [(25, 2048, 2048), (26, 2048, 2049), (30, 2049, 2048), (31, 2047, 2050)])
def test_gram_of_long_odd_rows(gpu, m, n2, n3):
    """25 to 31 rows on both sides of 2^22 columns.  FP32 products in chains of 64 are off by 65 u of the sum of their
    magnitudes at most, FP64 ones by nothing that shows: eigenvalues to 65 u of the trace."""
    import torch
    g = torch.Generator(device=gpu).manual_seed(m)
    x = torch.randn((n3, n2, m), generator=g, device=gpu) * torch.logspace(0, -2, m, device=gpu)
    a = x.reshape(-1, m)
    lam = sum(p.double().t() @ p.double() for p in a.split(1 << 20))
    want = torch.linalg.eigvalsh(lam).flip(0).cpu().numpy()
    got = np.asarray(_ttr().tt_svd(x.permute(2, 1, 0), [1, 4, 4, 1], gemm="fp32").sigmas[0][:m]) ** 2
    assert np.abs(got - want).max() <= 65 * U32 * want.sum()


@pytest.mark.parametrize("m,n,N", [(600, 200000, 96), (256, 600000, 80), (4096, 37000, 64), (600, 200000, 24),
                                   (130, 600000, 128)])
def test_sketch_fp32_chain_length(gpu, m, n, N):
    """FP32 sums of a sketch run over at most 1024 of these columns.  Products of 1 + 2^-14 add up exactly as long as
    the sum is below 1024 and lose 2^-14 each from there on; everything after the chains is FP64."""
    import torch
    a = torch.ones((n, m), device=gpu).t()
    w = torch.full((N, n), 1.0 + 2.0 ** -14, device=gpu).t()
    y = _ttr().sketch(a, w, "fp32")
    assert torch.all(y.double() == n * (1.0 + 2.0 ** -14))


@pytest.mark.parametrize("ring,n", [(False, (5, 3)), (False, (130, 70)), (False, (128, 64)), (False, (9, 15, 33, 7)),
                                    (True, (130, 3, 131)), (True, (16, 9, 17))])
def test_rel_error_of_an_infinite_core(gpu, ring, n):
    """Positive cores of rank 1 of which one entry is infinite: the reconstruction is infinite there and nowhere NaN,
    and so is the error, whatever the sizes leave of the last tiles."""
    rng = np.random.default_rng(sum(n))
    cores = [rng.uniform(0.5, 1.0, (1, k, 1)).astype(np.float32) for k in n]
    x = (oracle.tr_full if ring else oracle.tt_full)([c.astype(np.float64) for c in cores]).astype(np.float32)
    for k in (0, len(n) - 1):
        bad = [c.copy() for c in cores]
        bad[k][0, 1, 0] = np.inf
        assert _ttr().rel_error(_dev(x, gpu), [_dev(c, gpu) for c in bad], ring=ring) == np.inf


@pytest.mark.parametrize("ring,n,ranks", [
    (False, (2000, 10, 12, 14), (1, 5, 7, 4, 1)),
    (True, (700, 20, 30, 13), (3, 5, 7, 4, 3)),
    (True, (900, 10, 60, 2), (2, 5, 7, 4, 2)),
    (False, (1500, 12, 10, 8, 9), (1, 4, 8, 30, 9, 1)),
])
def test_rel_error_within_its_scratch(gpu, monkeypatch, ring, n, ranks):
    """A long first mode, so that every cut but the first would merge a larger left side than the cores right of it.
    The check takes two FP32 buffers of the largest of those, 1 MiB and 4 KiB of alignment, as its context allows here."""
    ttr = _ttr()
    rng = np.random.default_rng(sum(n))
    d = len(n)
    cores = [rng.standard_normal((ranks[k], n[k], ranks[k + 1])).astype(np.float32) for k in range(d)]
    full = (oracle.tr_full if ring else oracle.tt_full)([c.astype(np.float64) for c in cores])
    x = (full + 1e-2 * np.linalg.norm(full) / np.sqrt(full.size) * rng.standard_normal(n)).astype(np.float32)
    most = max(ranks[k] * int(np.prod(n[k:])) * ranks[d] for k in range(1, d))
    xd, cd = _dev(x, gpu), [_dev(c, gpu) for c in cores]
    want = oracle.rel_error(x, full)
    monkeypatch.setattr(ttr, "_CTX", {})
    assert ttr.lib().tt_ctx_set_alloc_limit(ttr._ctx_for(0), 8 * most + 4096 + (1 << 20)) == 0
    assert abs(ttr.rel_error(xd, cd, ring=ring) - want) <= 1e-9 * want


@pytest.mark.parametrize("ring,n,ranks,noise", [
    (False, (5, 3), (1, 3, 1), 1e-4),
    (False, (12, 12, 12, 12, 12), (1, 7, 40, 65, 9, 1), 1e-4),
    (False, (37, 29, 41, 23), (1, 19, 45, 13, 1), 1e-3),
    (True, (16, 9, 17, 8), (4, 3, 11, 2, 4), 1e-4),
    (True, (130, 3, 131), (2, 5, 6, 2), 1e-2),
])
def test_rel_error_is_fp64(gpu, ring, n, ranks, noise):
    """FP64 from the FP32 cores and X to the sums: at an error of `noise` the difference X - X^ holds 2^-53 x the sum of
    magnitudes / noise, 1e-9 of the result with room to spare; an FP32 X^ would move it by u / noise and more."""
    rng = np.random.default_rng(sum(n))
    d = len(n)
    cores = [rng.standard_normal((ranks[k], n[k], ranks[k + 1])).astype(np.float32) for k in range(d)]
    full = (oracle.tr_full if ring else oracle.tt_full)([c.astype(np.float64) for c in cores])
    x = (full + noise * np.linalg.norm(full) / np.sqrt(full.size) * rng.standard_normal(n)).astype(np.float32)
    want = oracle.rel_error(x, full)
    got = _ttr().rel_error(_dev(x, gpu), [_dev(c, gpu) for c in cores], ring=ring)
    assert abs(got - want) <= 1e-9 * want
