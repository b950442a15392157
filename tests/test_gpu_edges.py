"""Edge sizes of the FP32 / FP64 kernels: tile remainders, one-element sides, unaligned rows, and the
switch points of the launch rules, against NumPy in FP64."""
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


@pytest.mark.parametrize("ring,n,ranks", [
    (False, (5, 3), (1, 3, 1)),
    (False, (128, 128), (1, 32, 1)),              # one tile, one K chunk
    (False, (129, 127), (1, 33, 1)),              # remainders on every side
    (False, (4, 1, 260, 7), (1, 2, 2, 5, 1)),
    (False, (12, 12, 12, 12, 12), (1, 7, 40, 65, 9, 1)),
    (False, (6, 20, 20, 22), (1, 6, 64, 16, 1)),
    (True, (7, 6, 5), (3, 2, 4, 3)),
    (True, (16, 9, 17, 8), (4, 3, 11, 2, 4)),
    (True, (130, 3, 131), (2, 5, 6, 2)),
])
def test_rel_error_edges(gpu, ring, n, ranks):
    """FP32 products would be off by (sum of the bond sizes + order) u of the absolute sums, taken as 4x
    the sums themselves; FP64 ones are far inside."""
    rng = np.random.default_rng(sum(n))
    d = len(n)
    cores = [rng.standard_normal((ranks[k], n[k], ranks[k + 1])).astype(np.float32) for k in range(d)]
    full = (oracle.tr_full if ring else oracle.tt_full)([c.astype(np.float64) for c in cores])
    x = (full + 1e-2 * np.linalg.norm(full) / np.sqrt(full.size) * rng.standard_normal(n)).astype(np.float32)
    got = _ttr().rel_error(_dev(x, gpu), [_dev(c, gpu) for c in cores], ring=ring)
    q = ranks[0] if ring else 1
    assert abs(got - oracle.rel_error(x, full)) <= 4 * (sum(ranks) * q + d) * U32


@pytest.mark.parametrize("n,N", [(1, 1), (3, 3), (8, 8), (64, 9), (65, 17), (129, 40), (511, 33), (640, 127),
                                 (1471, 128), (60000, 129 - 1), (4097, 65)])
def test_cholqr2_edges(gpu, n, N):
    """Panel, row-chunk and cluster remainders; (60000, 128) takes the multi-launch path.  Two passes
    over a matrix of condition < 1e3: orthogonality is the FP32 rounding of Q's entries, u sqrt(n) per
    inner product of unit columns at worst, N^2 of them; Q R reproduces Y to the same."""
    import torch
    g = torch.Generator(device="cpu").manual_seed(n + N)
    y = torch.randn((N, n), generator=g).to(gpu).t()
    q, r = _ttr().cholqr2(y)
    qd, rd, yd = q.double().cpu().numpy(), r.cpu().numpy(), y.double().cpu().numpy()
    tol = 4 * U32 * N * max(1.0, np.sqrt(N))
    assert np.linalg.norm(qd.T @ qd - np.eye(N)) <= tol
    assert np.linalg.norm(qd @ rd - yd) <= tol * np.linalg.norm(yd)
    assert np.allclose(np.tril(rd, -1), 0.0) and np.all(np.diag(rd) > 0.0)
    q2, _ = _ttr().cholqr2(y, want_r=False)
    assert torch.equal(q, q2)  # R is a by-product: Q is the same with and without it


@pytest.mark.parametrize("n,N", [(1, 1), (3, 7), (31, 8), (33, 9), (1000, 17), (128, 32), (129, 33), (20000, 31),
                                 (65, 64), (40000, 65), (97, 128)])
@pytest.mark.parametrize("layout", ["col", "row", "strided"])
def test_gram_edges(gpu, n, N, layout):
    """Chunk, tile and group remainders in either layout, and rows inside a wider matrix: FP64 products
    of FP32 values are exact and the sums round at 2^-53 of the sum of magnitudes."""
    import ctypes as C
    import torch
    ttr = _ttr()
    rng = np.random.default_rng(n + N)
    wide = rng.standard_normal((n, N + 3)).astype(np.float32)
    z = torch.from_numpy(wide).to(gpu)
    if layout == "col":
        z = z[:, :N].t().contiguous()
        rs, cs = 1, n
    elif layout == "row":
        z = z[:, :N].contiguous()
        rs, cs = N, 1
    else:
        rs, cs = N + 3, 1
    w = torch.empty((N, N), dtype=torch.float64, device=gpu)
    ttr._lib.check(ttr.lib().tt_k_gram_tall(ttr._ctx_for(0), C.c_void_p(z.data_ptr()), n, N, rs, cs,
                                            C.c_void_p(w.data_ptr())))
    ref = wide[:, :N].astype(np.float64)
    bound = n * 2.0 ** -53 * (np.abs(ref).T @ np.abs(ref)) + 1e-300
    assert np.all(np.abs(w.cpu().numpy() - ref.T @ ref) <= 2 * bound)


@pytest.mark.parametrize("m", [1, 2, 3, 5, 6, 17, 30, 31])
@pytest.mark.parametrize("n", [1, 47, 48, 49, 100003])
def test_gram_rows_unaligned(gpu, m, n):
    """Unfoldings of up to 32 rows whose columns the TMA cannot address (through the decomposition's own
    rule: an exact step of tt_svd): sigma against NumPy."""
    import torch
    ttr = _ttr()
    rng = np.random.default_rng(m * n)
    a = rng.standard_normal((m, n)).astype(np.float32)
    r = min(m, n)
    res = ttr.tt_svd(_dev(a, gpu), [1, r, 1])
    ref = np.linalg.svd(a.astype(np.float64), compute_uv=False)
    # FP32 products and 64-term sums: the Gram is within 64 u of its entries' magnitudes
    tol = 64 * U32 * m * ref[0] ** 2
    assert np.all(np.abs(res.sigmas[0][:r].astype(np.float64) ** 2 - ref[:r] ** 2) <= tol)
    del torch


@pytest.mark.parametrize("m,n,N", [(1, 1, 1), (63, 9, 7), (64, 64, 16), (65, 63, 17), (100, 1000, 24), (129, 8, 40),
                                   (192, 100000, 33), (577, 4097, 41), (64, 513, 64), (66, 777, 65), (320, 640, 128)])
def test_sketch_fp32_edges(gpu, m, n, N):
    """Row tiles of 64, chunks of 8 columns dealt to 8 warps, column blocks above 64; rows that are not a
    multiple of 4.  A product-sum of n FP32 terms is off by at most n u of the sum of magnitudes; random
    signs leave about sqrt(n) of it, 8x that is allowed."""
    rng = np.random.default_rng(m + n + N)
    a, w = rng.standard_normal((m, n)).astype(np.float32), rng.standard_normal((n, N)).astype(np.float32)
    y = _ttr().sketch(_dev(a, gpu), _dev(w, gpu), "fp32").cpu().numpy()
    ref = a.astype(np.float64) @ w.astype(np.float64)
    bound = 8 * np.sqrt(n) * U32 * (np.linalg.norm(a, axis=1)[:, None] * np.linalg.norm(w, axis=0)[None, :])
    assert np.all(np.abs(y - ref) <= bound)


@pytest.mark.parametrize("m,n,N", [(65, 127, 5), (66, 128, 16), (67, 129, 17), (128, 1000, 24), (131, 400, 40),
                                   (600, 70, 57), (96, 300, 65), (1300, 20, 128), (68, 60000, 33),
                                   # up to 64 rows: the small-K kernel, one and several columns per thread
                                   (1, 5, 1), (30, 200000, 20), (33, 80000, 9), (64, 100000, 64), (48, 90000, 48),
                                   (24, 100001, 8), (63, 300, 32), (2, 77777, 3)])
def test_project_fp32_edges(gpu, m, n, N):
    rng = np.random.default_rng(m + n + N)
    a, q = rng.standard_normal((m, n)).astype(np.float32), rng.standard_normal((m, N)).astype(np.float32)
    y = _ttr().project(_dev(a, gpu), _dev(q, gpu), "fp32").cpu().numpy()
    ref = q.astype(np.float64).T @ a.astype(np.float64)
    bound = 8 * np.sqrt(m) * U32 * (np.linalg.norm(q, axis=0)[:, None] * np.linalg.norm(a, axis=0)[None, :])
    assert np.all(np.abs(y - ref) <= bound)


@pytest.mark.parametrize("rank", [1, 4, 9, 20, 32])
def test_batched_edges(gpu, rank):
    """Tensors of that rank without noise come back up to the rounding of FP32 chains: a step of a tensor with
    sides m x c multiplies along m or c, relative errors of that length u, taken as 8x."""
    shapes = [(32, 200), (33, 33), (31, 1000), (700, 32), (1, 9), (9, 1), (5, 3, 2), (200, 3),  # exact steps' limits
              (192, 40), (193, 40), (384, 37), (385, 37), (512, 33),                          # rows per pass of a sketch
              (7, 70, 33), (34, 16, 36), (13, 11, 17, 5), (2, 3, 2, 3, 2, 3)]
    for order in sorted({len(n) for n in shapes}):
        xs = []
        for k, n in enumerate(shapes):
            r = [1] + [min(rank, int(np.prod(n[:j])), int(np.prod(n[j:]))) for j in range(1, len(n))] + [1]
            if len(n) == order:
                xs.append(oracle.make_tt_tensor(list(n), r, 0.0, seed=100 * rank + k))
        for x, (cores, ranks, _) in zip(xs, _ttr().tt_svd_batched(xs, eps=0.0, rmax=rank)):
            err = oracle.rel_error(x, oracle.tt_full([c.double().cpu().numpy() for c in cores]))
            assert err <= 8 * (x.ndim - 1) * max(max(x.shape), 64) * U32, (x.shape, ranks, err)


@pytest.mark.parametrize("N", [3, 4, 6, 7, 8, 9, 13, 30, 34, 48, 62])
def test_syev_row_parts(gpu, N):
    """Rows of eigenvectors split over four warps: uneven splits, one pair per warp, fewer pairs than warps."""
    import torch
    rng = np.random.default_rng(N)
    q = np.linalg.qr(rng.standard_normal((N, N)))[0]
    w = (q * np.logspace(0, -4, N)) @ q.T
    ev, vec, _ = _ttr().syev(torch.from_numpy(w).to(gpu))
    ev, vec = ev.cpu().numpy(), vec.cpu().numpy()
    assert np.max(np.abs(ev - np.logspace(0, -4, N))) < 1e-11
    assert np.linalg.norm(w @ vec - vec * ev) < 1e-10 * N
    assert np.linalg.norm(vec.T @ vec - np.eye(N)) < 1e-12 * N


@pytest.mark.parametrize("width", [65, 66, 71, 72, 73, 80, 101, 127, 128])
def test_wide_sketch_singular_values(gpu, width):
    """A sketch of 65 to 128 columns of which 16 are kept goes through the subspace eigen-solver (rows padded to a
    multiple of 8).  FP32 chains along the 130 rows: 130 u of the largest singular value."""
    n, r = (130, 12, 11), 4
    rng = np.random.default_rng(width)
    cores = [rng.standard_normal((r, k, r)) for k in n]
    x = oracle.tr_full(cores)
    x = (x + 1e-5 * np.linalg.norm(x) / np.sqrt(x.size) * rng.standard_normal(x.shape)).astype(np.float32)
    res = _ttr().tr_svd(_dev(x, gpu), [r, r, 11, r], gemm="fp32", oversample=width - r * r, power_iters=1)
    ref = np.linalg.svd(np.reshape(x, (130, -1), order="F").astype(np.float64), compute_uv=False)
    assert np.all(np.abs(res.sigmas[0][:r * r] - ref[:r * r]) <= 130 * U32 * ref[0])


def test_batched_two_per_sm_same_bits(gpu):
    """A batch large enough for two tensors per SM (the kernel with fewer registers) gives the bits of a small one."""
    import torch
    rng = np.random.default_rng(11)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    xs = [rng.standard_normal(rng.integers(4, 40, size=3)).astype(np.float32) for _ in range(4 * sms + 8)]
    few, many = (_ttr().tt_svd_batched(x, eps=0.3, rmax=12) for x in (xs[:40], xs))
    for (c0, r0, e0), (c1, r1, e1) in zip(few, many):
        assert r0 == r1 and e0 == e1 and all(torch.equal(a, b) for a, b in zip(c0, c1))
