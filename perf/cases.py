"""The work this library is used for, as cases that can be timed and compared.

Five kinds, each through the package's public calls:

* ``tt``     one tensor to a tensor train at fixed ranks (``tt_svd``), device or host tensor;
* ``tr``     one tensor to a tensor ring at fixed bond ranks (``tr_svd``);
* ``eps``    one tensor to a tolerance, ranks found on the way, plain or learned (``tt_svd`` with eps);
* ``batch``  many small tensors through one plan (``Batch``), run again and again;
* ``check``  the way back: the reconstruction error of given cores (``rel_error``).

Tensors are built on the GPU from random N(0,1) cores plus relative Gaussian noise, as in the
repository's benchmark and tests.  A case holds plain values only: ``shape`` and ``ranks`` are texts
like "32x32x32".
"""
import math
import random

import numpy as np
import torch

import tensor_train_ring_decompositions_hpc_gpu_b200 as ttr
from tensor_train_ring_decompositions_hpc_gpu_b200 import learned

FP32_LIMIT = 1 << 24  # gemm "auto" keeps unfoldings below this many elements on the FP32 kernels


def _ints(text):
    return [int(v) for v in text.split("x")]


def _text(values):
    return "x".join(str(v) for v in values)


def _tt(name, shape, ranks, noise, gemm="auto", power=0, host=False):
    return {"name": name, "kind": "tt", "shape": shape, "ranks": ranks, "noise": noise, "gemm": gemm,
            "oversample": 8, "power": power, "host": host}


def listed():
    return [
        # a tensor of one small block of a larger computation: launches and latency are all of it
        _tt("tt4_16", "16x16x16x16", "1x8x8x8x1", 1e-4),
        # the plain third-order decomposition: 256^3, ranks 16, s = 8, one power iteration, FP32
        _tt("tt3_256_fp32", "256x256x256", "1x16x16x1", 1e-3, gemm="fp32", power=1),
        # measured data rarely has round sizes: odd modes and ranks, no alignment to rely on
        _tt("tt5_ragged", "37x29x41x23x31", "1x19x45x37x13x1", 1e-4, power=1),
        # order 6 at full FP32 precision with the customary s = 8, p = 1
        _tt("tt6_24_fp32", "24x24x24x24x24x24", "1x24x24x24x24x24x1", 1e-4, gemm="fp32", power=1),
        # the headline: a 4.3 GB order-6 tensor at ranks 32
        _tt("tt6_32", "32x32x32x32x32x32", "1x32x32x32x32x32x1", 1e-4),
        # a tensor in (pinned) host memory, cores wanted on the host: the drop-in call of a host program
        _tt("tt3_host", "256x192x224", "1x24x20x1", 1e-3, host=True),
        # third-order ring, the smallest order that has one
        {"name": "tr3_128", "kind": "tr", "shape": "128x96x80", "ranks": "4x4x16x4", "bond": 4, "noise": 1e-4,
         "gemm": "auto", "oversample": 8, "power": 1},
        # the order-6 ring: bond ranks 8 cut through a flat spectrum, so a wide sketch and one power iteration
        {"name": "tr6_32", "kind": "tr", "shape": "32x32x32x32x32x32", "ranks": "8x8x8x8x8x8x8", "bond": 8,
         "noise": 1e-4, "gemm": "auto", "oversample": 72, "power": 1},
        # a tolerance instead of ranks, sketch widths chosen by the shipped predictor
        {"name": "eps6_learned", "kind": "eps", "shape": "30x26x34x24x28x32", "ranks": "1x20x40x48x40x20x1",
         "noise": 1e-4, "eps": 1e-3, "rmax": 64, "learned": True},
        # thousands of small uneven tensors decomposed per step of an outer loop
        {"name": "batch4_4096", "kind": "batch", "count": 4096, "order": 4, "nmin": 8, "nmax": 32, "rmin": 2,
         "rmax": 16, "sizes": 1, "noise": 1e-3, "eps": 1e-2},
        # the accuracy check that follows a decomposition
        {"name": "check6_32", "kind": "check", "ring": False, "shape": "32x32x32x32x32x32",
         "ranks": "1x32x32x32x32x32x1", "noise": 1e-4},
    ]


def _draw_shape(rng, lo, hi, orders, nmin=6, nmax=400):
    """Mode sizes of a random order whose product is spread over the logarithm of [lo, hi]."""
    while True:
        d = rng.choice(orders)
        size = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        n = [int(round(size ** (1.0 / d) * math.exp(rng.uniform(-0.45, 0.45)))) for _ in range(d)]
        if all(nmin <= v <= nmax for v in n) and lo / 2 <= math.prod(n) <= hi:
            return n


def _draw_ranks(rng, n, cap):
    """TT ranks that a tensor with these modes carries with room to spare on both sides."""
    d, r = len(n), [1]
    for k in range(1, d):
        most = min(cap, 3 * r[-1] * n[k - 1] // 4, 3 * math.prod(n[k:]) // 4)
        r.append(rng.randint(2, max(2, most)))
    r.append(1)
    for k in range(d - 1, 0, -1):  # the same bound from the right
        r[k] = max(2, min(r[k], 3 * n[k] * r[k + 1] // 4))
    return r


def draw(rng: random.Random):
    kind = rng.choice(["tt", "tt", "tt", "tr", "eps", "batch", "check"])
    if kind == "tt":
        host = rng.random() < 0.15
        n = _draw_shape(rng, 4e3, 6e7 if host else 9e8, [3, 4, 5, 6])
        c = _tt("", _text(n), _text(_draw_ranks(rng, n, 48)), rng.choice([1e-4, 1e-3]),
                gemm=rng.choice(["auto", "auto", "fp32"]), power=rng.choice([0, 1]), host=host)
        del c["name"]
        return c
    if kind == "tr":
        n = _draw_shape(rng, 2e4, 5e8, [3, 4, 5, 6], nmin=8)
        b = rng.randint(2, max(2, min(5, math.isqrt(n[0]))))
        r = [b, b]
        for k in range(2, len(n)):
            r.append(min(b * b, r[-1] * n[k - 1], math.prod(n[k:]) * b))
        return {"kind": "tr", "shape": _text(n), "ranks": _text(r + [b]), "bond": b, "noise": 1e-4,
                "gemm": rng.choice(["auto", "auto", "fp32"]), "oversample": 8, "power": rng.choice([0, 1])}
    if kind == "eps":
        n = _draw_shape(rng, 1e6, 6e8, [4, 5, 6], nmin=10)
        return {"kind": "eps", "shape": _text(n), "ranks": _text(_draw_ranks(rng, n, 40)), "noise": 1e-4,
                "eps": 1e-3, "rmax": 64, "learned": rng.random() < 0.5}
    if kind == "batch":
        lo = rng.randint(5, 12)
        return {"kind": "batch", "count": int(round(math.exp(rng.uniform(math.log(64), math.log(3000))))),
                "order": rng.choice([3, 4, 4]), "nmin": lo, "nmax": rng.randint(lo + 4, 32), "rmin": 2,
                "rmax": rng.randint(6, 16), "sizes": rng.randrange(1 << 20), "noise": 1e-3, "eps": 1e-2}
    ring = rng.random() < 0.4
    n = _draw_shape(rng, 1e5, 9e8, [3, 4, 5, 6])
    r = [rng.randint(2, 6)] * (len(n) + 1) if ring else _draw_ranks(rng, n, 32)
    return {"kind": "check", "ring": ring, "shape": _text(n), "ranks": _text(r), "noise": 1e-4}


# ---- inputs ----
def _logical(flat, shape):
    """The tensor (i1, ..., id) whose column-major storage is ``flat``."""
    d = len(shape)
    return flat.view(*reversed(shape)).permute(*reversed(range(d)))


def _random_cores(shape, ranks, gen):
    return [torch.randn(ranks[k], shape[k], ranks[k + 1], generator=gen, device="cuda") for k in range(len(shape))]


def _contract(cores):
    """Column-major flat tensor of a train or a ring (first and last ranks are equal)."""
    if cores[0].shape[0] == 1:
        t = cores[-1][:, :, 0].t().contiguous()  # (i_d, a)
        for c in reversed(cores[:-1]):
            r0, n, r1 = c.shape
            t = (t @ c.permute(2, 1, 0).reshape(r1, n * r0)).reshape(-1, r0)
        return t.reshape(-1)
    m = cores[-1].permute(2, 1, 0)  # (a0, i_d, b)
    for c in reversed(cores[1:-1]):
        r0, n, r1 = c.shape
        m = (m @ c.permute(2, 1, 0).reshape(r1, n * r0)).reshape(m.shape[0], -1, r0)
    a, rest, b = m.shape  # X[J, i1] = sum m[a, J, b] G1[a, i1, b]
    return (m.permute(1, 0, 2).reshape(rest, a * b) @ cores[0].permute(0, 2, 1).reshape(a * b, -1)).reshape(-1)


def _add_noise(x, rel, gen):
    scale = rel * float(torch.linalg.vector_norm(x, dtype=torch.float64)) / math.sqrt(x.numel())
    for part in x.split(1 << 28):
        part.add_(torch.randn(part.shape, generator=gen, device="cuda"), alpha=scale)
    return x


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _tensor(case, seed):
    """(column-major flat tensor, the cores it was made from)."""
    gen = _generator(seed)
    shape, ranks = _ints(case["shape"]), _ints(case["ranks"])
    if case["kind"] == "tr":
        ranks = [case["bond"]] * (len(shape) + 1)
    cores = _random_cores(shape, ranks, gen)
    return _add_noise(_contract(cores), case["noise"], gen), cores


def _small_tensors(case, seed):
    """Tensors whose sizes and ranks come with the case (``sizes`` seeds them), the values with the seed."""
    rng, gen = random.Random(case["sizes"]), _generator(seed)
    d, total, specs = case["order"], 0, []
    for _ in range(case["count"]):
        n = [rng.randint(case["nmin"], case["nmax"]) for _ in range(d)]
        r = [1] + [rng.randint(case["rmin"], case["rmax"]) for _ in range(d - 1)] + [1]
        need = sum(r[k] * n[k] * r[k + 1] for k in range(d))
        specs.append((n, r, total))
        total += need
    values = torch.randn(total, generator=gen, device="cuda")
    out = []
    for n, r, off in specs:
        cores = []
        for k in range(d):
            need = r[k] * n[k] * r[k + 1]
            cores.append(values[off:off + need].view(r[k], n[k], r[k + 1]))
            off += need
        x = _contract(cores)
        x = x + (case["noise"] / math.sqrt(x.numel())) * torch.linalg.vector_norm(x) * torch.randn(
            x.shape, generator=gen, device="cuda")
        out.append(_logical(x, n))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = ttr.Batch(_small_tensors(case, seed), rmax=case["rmax"])
        b.make_plan(eps=case["eps"])
        return {"kind": kind, "batch": b, "eps": case["eps"]}
    shape, ranks = _ints(case["shape"]), _ints(case["ranks"])
    x, cores = _tensor(case, seed)
    state = {"kind": kind, "x": _logical(x, shape), "ranks": ranks}
    if kind == "check":
        state.update(cores=cores, ring=case["ring"])
        return state
    if kind == "eps":
        ttr.set_predictor(learned.load_params())
        state["ranks"] = [1] + [case["rmax"]] * (len(shape) - 1) + [1]
        state["options"] = {"eps": case["eps"], "power_iters": 1,
                            "flags": ttr.TT_FLAG_LEARNED if case["learned"] else ttr.TT_FLAG_ADAPTIVE_KS}
        return state
    state["options"] = {"gemm": case["gemm"], "oversample": case["oversample"], "power_iters": case["power"]}
    if case.get("host"):
        pinned = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
        pinned.copy_(x)
        state.update(x=pinned.numpy().reshape(shape, order="F"), pinned=pinned)
    return state


# ---- one pass ----
def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        b.run(eps=state["eps"])
        return {"cores": b.cores, "ranks": np.array(b.ranks), "err": np.array(b.err, dtype=np.float32)}
    if kind == "check":
        return ttr.rel_error(state["x"], state["cores"], ring=state["ring"])
    res = (ttr.tr_svd if kind == "tr" else ttr.tt_svd)(state["x"], state["ranks"], **state["options"])
    # the singular values that the decomposition keeps, in the precision the library reports them
    r = res.ranks
    kept = [r[0] * r[1] if kind == "tr" else r[1]] + r[2:-1]
    out = {"cores": res.cores, "sigma": [s[:k].astype(np.float32) for s, k in zip(res.sigmas, kept)]}
    if kind == "eps":
        out["ranks"] = np.array(r)
    return out


# ---- the work it cannot do without ----
def work(case):
    """Bytes: every input read once, every output written once.  FLOPs: each unfolding of the chain
    multiplied twice by a matrix of its target rank (once to find the basis, once to project on it)."""
    if case["kind"] == "batch":
        n, r, d = (case["nmin"] + case["nmax"]) / 2, (case["rmin"] + case["rmax"]) / 2, case["order"]
        core = case["count"] * (2 * n * r + (d - 2) * n * r * r)
        size = case["count"] * n ** d
        flops = sum(4.0 * size * r / (1 if k == 0 else n ** k / r) for k in range(d - 1))
        return {"bytes": 4.0 * (size + core), "flops": flops}
    shape, ranks = _ints(case["shape"]), _ints(case["ranks"])
    d, size = len(shape), math.prod(shape)
    core = sum(ranks[k] * shape[k] * ranks[k + 1] for k in range(d))
    if case["kind"] == "check":
        return {"bytes": 4.0 * (size + core), "flops": 2.0 * size * ranks[0] * ranks[1]}
    flops, rest = 0.0, size
    for k in range(d - 1):
        q = ranks[0] * ranks[1] if k == 0 and case["kind"] == "tr" else ranks[k + 1]
        rows = (1 if k == 0 else ranks[k]) * shape[k]
        cols = rest // shape[k] * (ranks[0] if k > 0 and case["kind"] == "tr" else 1)
        q = min(q, rows, cols)
        flops += 4.0 * rows * cols * q
        rest //= shape[k]
    return {"bytes": 4.0 * (size + core), "flops": flops}


# ---- the same in 64 bits ----
def _basis(a, r):
    """Leading r left singular vectors of ``a`` (largest entry of each made positive) and all singular values."""
    m, n = a.shape
    if m <= n:
        lam, u = torch.linalg.eigh(a @ a.t())
        sig, u = lam.flip(0).clamp_min(0).sqrt(), u.flip(1)[:, :r]
    else:
        lam, v = torch.linalg.eigh(a.t() @ a)
        sig = lam.flip(0).clamp_min(0).sqrt()
        u = a @ v.flip(1)[:, :r] / sig[:r]
    u = u * torch.sign(u.gather(0, u.abs().argmax(0, keepdim=True)))
    return u, sig


def _exact_chain(x, shape, ranks, ring):
    """Cores and kept singular values of the truncated chain.  A step that keeps every row leaves the
    data as it is and hands its rotation to the next core, so that signs are those of the library."""
    d, data, cores, sigma = len(shape), x.double(), [], []
    rows, pending = 1, None
    for k in range(d - 1):
        q = ranks[0] * ranks[1] if ring and k == 0 else ranks[k + 1]
        a = data.view(-1, rows * shape[k]).t()
        u, sig = _basis(a, min(q, *a.shape))
        sigma.append(sig[:q])
        core = u.t().reshape(-1, shape[k], rows)  # (b, i, a)
        if pending is not None:
            core = core @ pending
        if ring and k == 0:
            r0 = ranks[0]
            r1 = -(-u.shape[1] // r0)
            full = torch.zeros(r0 * ranks[1], shape[0], dtype=u.dtype, device=u.device)
            full[:u.shape[1]] = u.t()
            cores.append(full.view(ranks[1], r0, shape[0]).permute(1, 2, 0))
            y = torch.zeros(a.shape[1], r0 * r1, dtype=u.dtype, device=u.device)
            y[:, :u.shape[1]] = a.t() @ u
            data = y.view(-1, r1, r0).permute(2, 0, 1).reshape(-1)
            rows = r1
            continue
        cores.append(core.permute(2, 1, 0))
        if q == a.shape[0] and a.shape[0] <= a.shape[1] and not ring:
            pending = u
        else:
            data, pending = (a.t() @ u).reshape(-1), None
        rows = u.shape[1]
    last = data.view(-1, shape[-1], rows)
    cores.append((last if pending is None else last @ pending).permute(2, 1, 0))
    return cores, sigma


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":  # some 10^4 decompositions one by one: too long
        return None
    shape, ranks = _ints(case["shape"]), _ints(case["ranks"])
    x, made_from = _tensor(case, seed)
    if kind == "check":
        num = den = 0.0
        back = _contract([c.double() for c in made_from])
        for p, q in zip(x.split(1 << 28), back.split(1 << 28)):
            num += float((p.double() - q).square().sum())
            den += float(p.double().square().sum())
        return math.sqrt(num / den)
    if kind == "eps":  # the ranks are the tensor's own: far above the tolerance, the noise far below it
        cores, sigma = _exact_chain(x, shape, ranks, False)
        return {"cores": None, "sigma": [s.cpu().numpy() for s in sigma], "ranks": None}
    cores, sigma = _exact_chain(x, shape, ranks, kind == "tr")
    # A basis has an exact value where rounding alone stands between it and the library's: FP32
    # products, a power iteration between the sketch and the noise, and a clear gap below the rank
    # (a ring's later unfoldings are cut through a flat spectrum).
    fp32 = case["gemm"] == "fp32" or x.numel() < FP32_LIMIT
    return {"cores": cores if fp32 and case["power"] > 0 and kind == "tt" else [None] * len(cores),
            "sigma": [s.cpu().numpy() for s in sigma]}
