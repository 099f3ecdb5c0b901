"""Performance cases of the library: what a program that solves symmetric
positive definite systems with it has it do, through the public entry points
(``dplasma_b200.Context`` and ``dplasma_b200.autograd``).

``listed()`` names the standard cases, ``draw(rng)`` gives one more of the same
ranges, ``prepare`` makes what a program holds before the call, ``run`` is one
pass, ``exact`` the same result in plain torch at 64 bits.

The calls that factor in place overwrite their matrix, so a pass first copies
the matrix (and right-hand sides) from the program's own copy, as a program
that factors a new matrix of the same shape on each pass does.
"""
import math
import random

import torch

import dplasma_b200 as db
from dplasma_b200 import autograd as dag

F64 = torch.float64
EPS = 2.0 ** -53
UPLO = {"L": db.Lower, "U": db.Upper}
FMT = {"fp16": db.FP16, "bf16": db.BF16, "split": db.FP16_SPLIT}
REFLECTORS = 32                 # of the conditioned matrices


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest dense call: the size and ragged tile of the tester's quick configuration
        {"name": "posv_378", "kind": "posv", "n": 378, "nb": 93, "uplo": "L", "layout": "tile", "nrhs": 4},
        # one ordinary factor-and-solve of a matrix that lives in device tiles
        {"name": "posv_4096", "kind": "posv", "n": 4096, "nb": 256, "uplo": "L", "layout": "tile", "nrhs": 64},
        # a column-major caller's upper factor, the order no multiple of the tile
        {"name": "potrf_7000_upper", "kind": "potrf", "n": 7000, "nb": 320, "uplo": "U", "layout": "lapack"},
        # the large plain FP64 factorization, bound by arithmetic
        {"name": "potrf_32768", "kind": "potrf", "n": 32768, "nb": 512, "uplo": "L", "layout": "tile"},
        # solves on a factor that is kept (time stepping, many right-hand sides one after the other)
        {"name": "potrs_16384", "kind": "potrs", "n": 16384, "nb": 256, "uplo": "L", "layout": "tile", "nrhs": 16},
        # mixed precision with refinement to FP64 accuracy: well conditioned, plain FP16 operands
        {"name": "sposv_12288_fp16", "kind": "sposv", "n": 12288, "nb": 256, "nrhs": 1, "kappa": 1e2, "fmt": "fp16"},
        # mixed precision at the library's headline size: ill conditioned, split operands
        {"name": "sposv_65536_split", "kind": "sposv", "n": 65536, "nb": 256, "nrhs": 16, "kappa": 1e6, "fmt": "split"},
        # thousands of small systems of uneven sizes: factor, solve, log-determinant
        {"name": "batched_f64", "kind": "batched", "count": 4096, "lo": 32, "hi": 512, "dtype": "f64", "nrhs": 1,
         "sizes": 11},
        # the same in single precision at the small end
        {"name": "batched_f32_small", "kind": "batched", "count": 8192, "lo": 8, "hi": 96, "dtype": "f32", "nrhs": 1,
         "sizes": 12},
        # a training step's likelihoods of many independent Gaussian processes, with gradients
        {"name": "gp_batch", "kind": "gp_batch", "count": 1024, "lo": 64, "hi": 256, "sizes": 13},
        # a differentiable Cholesky factor, forward and backward for a dense gradient of the factor
        {"name": "cholesky_grad_4096", "kind": "cholesky", "n": 4096},
        # one Gaussian process of an odd size: likelihood and gradients (factor, solve, inverse)
        {"name": "gp_6001", "kind": "gp", "n": 6001},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["posv", "posv", "potrf", "potrf", "potrs", "sposv", "sposv", "batched", "batched", "gp_batch",
                       "cholesky", "gp"])
    nb = rng.choice([93, 128, 192, 256, 256, 320, 384, 512])
    uplo, layout = rng.choice("LU"), rng.choice(["tile", "tile", "lapack"])
    if kind == "posv":
        return {"kind": kind, "n": _log_int(rng, 100, 12000), "nb": nb, "uplo": uplo, "layout": layout,
                "nrhs": _log_int(rng, 1, 64)}
    if kind == "potrf":
        n = _log_int(rng, 500, 30000)
        if rng.random() < 0.5:                                   # whole tiles: factored where it lies
            n = max(nb, n // nb * nb)
        return {"kind": kind, "n": n, "nb": nb, "uplo": uplo, "layout": layout}
    if kind == "potrs":
        return {"kind": kind, "n": _log_int(rng, 500, 24000), "nb": nb, "uplo": uplo, "layout": layout,
                "nrhs": _log_int(rng, 1, 32)}
    if kind == "sposv":
        fmt, kappa = rng.choice([("fp16", 1e2), ("bf16", 1e2), ("split", 1e4), ("split", 1e6)])
        n = _log_int(rng, 1000, 40000)
        if rng.random() < 0.7:
            n = max(256, n // 256 * 256)
        return {"kind": kind, "n": n, "nb": 256, "nrhs": _log_int(rng, 1, 16), "kappa": kappa, "fmt": fmt}
    if kind == "batched":
        lo = _log_int(rng, 4, 128)
        return {"kind": kind, "count": _log_int(rng, 64, 4096), "lo": lo, "hi": _log_int(rng, lo, 512),
                "dtype": rng.choice(["f64", "f64", "f32"]), "nrhs": rng.choice([1, 1, 4]), "sizes": rng.randrange(10 ** 6)}
    if kind == "gp_batch":
        lo = _log_int(rng, 8, 128)
        return {"kind": kind, "count": _log_int(rng, 32, 1024), "lo": lo, "hi": _log_int(rng, lo, 256),
                "sizes": rng.randrange(10 ** 6)}
    if kind == "cholesky":
        return {"kind": kind, "n": _log_int(rng, 100, 8000)}
    return {"kind": "gp", "n": _log_int(rng, 200, 10000)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_context = {}


def _ctx():
    """the program's library context (one GPU, one stream, its workspaces)"""
    if "c" not in _context:
        _context["c"] = db.Context(torch.cuda.current_device())
    return _context["c"]


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + salt) % (2 ** 63))


def _rand(shape, gen):
    return torch.rand(shape, dtype=F64, device="cuda", generator=gen).sub_(0.5)


def _stored(nt, uplo):
    """tiles of the stored triangle in storage order (packed tile columns)"""
    if uplo == "L":
        return [(m, n) for n in range(nt) for m in range(n, nt)]
    return [(m, n) for n in range(nt) for m in range(n + 1)]


def _matrix(case, seed):
    """Storage of a symmetric matrix, entries uniform in [-0.5, 0.5] and n added
    to the diagonal (what the library's own generator makes for its testers):
    a flat tile buffer of the stored triangle, or one column-major array."""
    n, nb, uplo = case["n"], case["nb"], case["uplo"]
    gen = _gen(seed, 1)
    if case["layout"] == "lapack":
        a = _rand((n, n), gen)
        a.diagonal().add_(n)
        return a.reshape(-1)
    nt = -(-n // nb)
    tiles = _rand((nt * (nt + 1) // 2, nb, nb), gen)
    for i, (m, c) in enumerate(_stored(nt, uplo)):
        if m == c:
            tiles[i].diagonal().add_(n)
    return tiles.reshape(-1)


def _desc(case, buf):
    n, nb = case["n"], case["nb"]
    if case["layout"] == "lapack":
        return db.attach(db.desc_general(n, n, nb, nb, storage=db.STORAGE_LAPACK, lda=n), buf)
    return db.attach(db.desc_sym(n, nb, UPLO[case["uplo"]]), buf)


def _rhs_desc(n, nb, nrhs, buf):
    return db.attach(db.desc_general(n, nrhs, nb, nb, storage=db.STORAGE_LAPACK, lda=n), buf)


def _conditioned(n, nb, kappa, seed):
    """Lower tiles of A = Q diag(s) Q^T, s geometric from 1 to kappa, Q the
    product of random Householder reflectors in compact form I - V T V^T, and
    (s, V, T)."""
    gen = _gen(seed, 2)
    k = min(REFLECTORS, n)
    s = torch.exp(torch.linspace(0.0, math.log(kappa), n, dtype=F64, device="cuda"))
    V = torch.randn((n, k), dtype=F64, device="cuda", generator=gen)
    V /= V.norm(dim=0, keepdim=True)
    G = V.t() @ V
    T = torch.zeros((k, k), dtype=F64, device="cuda")
    for i in range(k):
        T[i, i] = 2.0
        if i:
            T[:i, i] = -2.0 * (T[:i, :i] @ G[:i, i])
    # A = D - U1 (V T)^T - (V T) U1^T + (V T) M (V T)^T,  U1 = D V, M = V^T D V
    VT = V @ T
    U1 = s[:, None] * V
    M = V.t() @ U1
    Y = VT @ (0.5 * M) - U1                                       # A = D + VT Y^T + Y VT^T
    nt = -(-n // nb)
    pad = nt * nb - n
    L = torch.nn.functional.pad(torch.cat([VT, Y], 1), (0, 0, 0, pad))
    R = torch.nn.functional.pad(torch.cat([Y, VT], 1), (0, 0, 0, pad))
    sp = torch.nn.functional.pad(s, (0, pad))
    tiles = torch.empty((nt * (nt + 1) // 2, nb, nb), dtype=F64, device="cuda")
    at = 0
    for c in range(nt):
        rows = nt - c
        blk = R[c * nb:(c + 1) * nb] @ L[c * nb:].t()             # (column, row)
        tiles[at:at + rows] = blk.view(nb, rows, nb).transpose(0, 1)
        tiles[at].diagonal().add_(sp[c * nb:(c + 1) * nb])
        at += rows
    return tiles.reshape(-1), (s, V, T)


def _sizes(case):
    r = random.Random(case["sizes"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["count"])]


def _se_kernel(n, gen, nugget):
    x = torch.rand((n, 3), dtype=F64, device="cuda", generator=gen)
    k = torch.exp(torch.cdist(x, x).square_().mul_(-1.0 / (2 * 0.2 ** 2)))
    k = torch.triu(k) + torch.triu(k, 1).t()
    k.diagonal().add_(nugget)
    return k


def _kernels(case, seed, dtype, nugget):
    """squared-exponential kernel matrices of random points, one after the
    other in one flat buffer, and the targets"""
    sizes = _sizes(case)
    gen = _gen(seed, 3)
    flat = torch.empty(sum(n * n for n in sizes), dtype=dtype, device="cuda")
    at = 0
    for lo in range(0, len(sizes), 256):                          # many small matrices: padded groups
        group = sizes[lo:lo + 256]
        m = max(group)
        x = torch.rand((len(group), m, 3), dtype=F64, device="cuda", generator=gen)
        d2 = (x[:, :, None, :] - x[:, None, :, :]).square_().sum(-1)
        k = torch.exp(d2.mul_(-1.0 / (2 * 0.2 ** 2)))
        k.diagonal(dim1=1, dim2=2).add_(nugget)
        for i, n in enumerate(group):
            flat[at:at + n * n].view(n, n).copy_(k[i, :n, :n])
            at += n * n
    y = torch.randn(sum(sizes), dtype=F64, device="cuda", generator=gen).to(dtype)
    return sizes, flat, y


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "ctx": _ctx()}
    if kind in ("posv", "potrf", "potrs"):
        n, nb = case["n"], case["nb"]
        st["A0"] = _matrix(case, seed)
        st["A"] = st["A0"].clone()
        st["dA"] = _desc(case, st["A"])
        if kind != "potrf":
            st["B0"] = _rand((case["nrhs"] * n,), _gen(seed, 4))
            st["B"] = st["B0"].clone()
            st["dB"] = _rhs_desc(n, nb, case["nrhs"], st["B"])
        if kind == "potrs":                                       # the factor that the program keeps
            db.torch_ready(st["A"])
            if st["ctx"].dpotrf(UPLO[case["uplo"]], st["dA"]) != 0:
                raise RuntimeError(st["ctx"].last_error())
            del st["A0"]
    elif kind == "sposv":
        n, nb, nrhs = case["n"], case["nb"], case["nrhs"]
        st["A"], _ = _conditioned(n, nb, case["kappa"], seed)
        st["dA"] = db.attach(db.desc_sym(n, nb, db.Lower), st["A"])
        st["B"] = _rand((nrhs * n,), _gen(seed, 4))
        st["X"] = torch.zeros_like(st["B"])
        st["dB"], st["dX"] = _rhs_desc(n, nb, nrhs, st["B"]), _rhs_desc(n, nb, nrhs, st["X"])
    elif kind == "batched":
        dt = F64 if case["dtype"] == "f64" else torch.float32
        sizes, st["K0"], y = _kernels(case, seed, dt, 1e-4 if dt == F64 else 1e-1)
        nrhs = case["nrhs"]
        st["y0"] = torch.cat([v.repeat(nrhs) for v in torch.split(y, sizes)]) if nrhs > 1 else y
        st["K"], st["y"] = st["K0"].clone(), st["y0"].clone()
        st["dt"] = dt
        st["n"] = torch.tensor(sizes, dtype=torch.int32, device="cuda")
        nn = torch.tensor(sizes, dtype=torch.int64, device="cuda")
        es = st["K"].element_size()
        st["pA"] = st["K"].data_ptr() + es * (torch.cumsum(nn * nn, 0) - nn * nn)
        st["pB"] = st["y"].data_ptr() + es * nrhs * (torch.cumsum(nn, 0) - nn)
        st["logdet"] = torch.empty(len(sizes), dtype=F64, device="cuda")
        st["info"] = torch.empty(len(sizes), dtype=torch.int32, device="cuda")
    elif kind == "gp_batch":
        st["sizes"], K, y = _kernels(case, seed, F64, 1e-4)
        st["K"], st["y"] = K.requires_grad_(True), y.requires_grad_(True)
    elif kind == "cholesky":
        n = case["n"]
        st["K"] = _se_kernel(n, _gen(seed, 5), 1e-2).requires_grad_(True)
        st["G"] = _rand((n, n), _gen(seed, 6)).tril_()
    elif kind == "gp":
        n = case["n"]
        st["K"] = _se_kernel(n, _gen(seed, 5), 1e-2).requires_grad_(True)
        st["y"] = torch.randn(n, dtype=F64, device="cuda", generator=_gen(seed, 6)).requires_grad_(True)
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _done(st, rc):
    if rc != 0:
        raise RuntimeError("%s: %d %s" % (st["case"]["kind"], rc, st["ctx"].last_error()))


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "posv":
        st["A"].copy_(st["A0"])
        st["B"].copy_(st["B0"])
        db.torch_ready(st["A"], st["B"])
        _done(st, ctx.dposv(UPLO[case["uplo"]], st["dA"], st["dB"]))
        return {"A": st["A"], "X": st["B"]}
    if kind == "potrf":
        st["A"].copy_(st["A0"])
        db.torch_ready(st["A"])
        _done(st, ctx.dpotrf(UPLO[case["uplo"]], st["dA"]))
        return {"A": st["A"]}
    if kind == "potrs":
        st["B"].copy_(st["B0"])
        db.torch_ready(st["B"])
        _done(st, ctx.dpotrs(UPLO[case["uplo"]], st["dA"], st["dB"]))
        return {"X": st["B"]}
    if kind == "sposv":
        db.torch_ready(st["B"])
        rc, stats = ctx.dsposv(db.Lower, st["dA"], st["dB"], st["dX"], fmt=FMT[case["fmt"]])
        _done(st, rc)
        return {"X": st["X"], "fallback": int(stats["fallback"])}
    if kind == "batched":
        st["K"].copy_(st["K0"])
        st["y"].copy_(st["y0"])
        _done(st, ctx.posv_batched_arrays(st["dt"], case["count"], st["n"], st["n"], st["pA"], st["pB"], case["nrhs"],
                                          st["logdet"], st["info"]))
        return {"K": st["K"], "x": st["y"], "logdet": st["logdet"], "info": st["info"]}
    if kind == "gp_batch":
        v = dag.gp_log_marginal_likelihood_flat(st["K"], st["y"], st["sizes"])
        dK, dy = torch.autograd.grad(v.sum(), (st["K"], st["y"]))
        return {"value": v.detach(), "dK": dK, "dy": dy}
    if kind == "cholesky":
        L = dag.cholesky(st["K"])
        (dK,) = torch.autograd.grad(L, st["K"], st["G"])
        return {"L": L.detach(), "dK": dK}
    v = dag.gp_log_marginal_likelihood(st["K"], st["y"])
    dK, dy = torch.autograd.grad(v, (st["K"], st["y"]))
    return {"value": v.detach(), "dK": dK, "dy": dy}


# ---------------------------------------------------------------------------
# work and tolerances
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("batched", "gp_batch"):
        sizes = _sizes(case)
        nrhs = case.get("nrhs", 1)
        es = 4 if case.get("dtype") == "f32" else 8
        if kind == "batched":
            return {"flops": sum(n ** 3 / 3 + 2 * n * n * nrhs for n in sizes),
                    "bytes": es * sum(n * (n + 1) + 2 * n * nrhs for n in sizes)}
        # factor and solve, then the inverse from the factor; the kernel read and its gradient written
        return {"flops": sum(n ** 3 + 2 * n * n for n in sizes), "bytes": es * sum(2 * n * n + 2 * n for n in sizes)}
    n = case["n"]
    nrhs = case.get("nrhs", 0)
    tri = n * (n + 1) / 2
    if kind == "posv":
        return {"flops": n ** 3 / 3 + 2 * n * n * nrhs, "bytes": 8 * (2 * tri + 2 * n * nrhs)}
    if kind == "potrf":
        return {"flops": n ** 3 / 3, "bytes": 8 * 2 * tri}
    if kind in ("potrs", "sposv"):
        return {"flops": (n ** 3 / 3 if kind == "sposv" else 0) + 2 * n * n * nrhs, "bytes": 8 * (tri + 2 * n * nrhs)}
    if kind == "cholesky":
        # factor; backward: the triangular inverse and three products that keep to the triangles
        return {"flops": n ** 3 / 3 + 4 * n ** 3 / 3, "bytes": 8 * (2 * tri + 2 * tri + n * n)}
    return {"flops": n ** 3 + 2 * n * n, "bytes": 8 * (tri + n * n + 3 * n)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("posv", "potrf"):
        # well conditioned: a few roundings of 64-bit sums (measured 1e-16 .. 9e-16)
        return {"rel": 5e-15}
    if kind == "potrs":
        return {"rel": 2e-14}                                     # measured 3e-15 .. 4e-15
    if kind == "sposv":
        # the stopping test bounds the residual by eps sqrt(n) |A| |x|, the error by kappa times that
        return {"rel": 4 * case["kappa"] * EPS * math.sqrt(case["n"])}
    # kernel matrices: the rounding times a condition of about order / nugget
    # (measured: solutions 9e-12 at 64 bits and 9e-7 at 32, gradients 4e-12)
    if kind == "batched":
        return {"rel": 5e-11} if case["dtype"] == "f64" else {"rel": 3e-5}
    return {"rel": 5e-11}


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _dense(case, buf):
    """the symmetric matrix of a storage buffer"""
    n, nb, uplo = case["n"], case["nb"], case["uplo"]
    if case["layout"] == "lapack":
        a = buf.view(n, n).t()                                    # column-major
        return torch.tril(a) + torch.tril(a, -1).t() if uplo == "L" else torch.triu(a) + torch.triu(a, 1).t()
    nt = -(-n // nb)
    tiles = buf.view(-1, nb, nb)
    a = torch.zeros((nt * nb, nt * nb), dtype=F64, device="cuda")
    for i, (m, c) in enumerate(_stored(nt, uplo)):
        a[m * nb:(m + 1) * nb, c * nb:(c + 1) * nb] = tiles[i].t()
    a = a[:n, :n]
    return torch.tril(a) + torch.tril(a, -1).t() if uplo == "L" else torch.triu(a) + torch.triu(a, 1).t()


def _with_factor(case, buf, L):
    """the storage buffer with the factor in the caller's triangle, all else as it was"""
    n, nb, uplo = case["n"], case["nb"], case["uplo"]
    out = buf.clone()
    if case["layout"] == "lapack":
        a = out.view(n, n)                                        # row r of the view = column r
        if uplo == "L":
            a.copy_(torch.triu(L.t()) + torch.tril(a, -1))
        else:
            a.copy_(torch.tril(L) + torch.triu(a, 1))
        return out
    nt = -(-n // nb)
    tiles = out.view(-1, nb, nb)
    for i, (m, c) in enumerate(_stored(nt, uplo)):
        rm, cm = min(nb, n - m * nb), min(nb, n - c * nb)
        # (column, row) view of the tile
        if uplo == "L":
            f = L[m * nb:m * nb + rm, c * nb:c * nb + cm].t()
            tiles[i, :cm, :rm] = torch.triu(f) + torch.tril(tiles[i, :cm, :rm], -1) if m == c else f
        else:
            f = L[c * nb:c * nb + cm, m * nb:m * nb + rm]
            tiles[i, :cm, :rm] = torch.tril(f) + torch.triu(tiles[i, :cm, :rm], 1) if m == c else f
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("posv", "potrf", "potrs"):
        n = case["n"]
        buf = _matrix(case, seed)
        L = torch.linalg.cholesky(_dense(case, buf))
        out = {}
        if kind != "potrs":
            out["A"] = _with_factor(case, buf, L)
        if kind != "potrf":
            b = _rand((case["nrhs"] * n,), _gen(seed, 4)).view(case["nrhs"], n).t()
            out["X"] = torch.cholesky_solve(b, L).t().reshape(-1)
        return out
    if kind == "sposv":
        n, nrhs = case["n"], case["nrhs"]
        _, (s, V, T) = _conditioned(n, case["nb"], case["kappa"], seed)
        b = _rand((nrhs * n,), _gen(seed, 4)).view(nrhs, n).t()
        # x = Q diag(1/s) Q^T b with Q = I - V T V^T
        y = (b - V @ (T.t() @ (V.t() @ b))) / s[:, None]
        x = y - V @ (T @ (V.t() @ y))
        return {"X": x.t().reshape(-1), "fallback": None}
    if kind == "batched":
        f64 = case["dtype"] == "f64"
        sizes, K, y = _kernels(case, seed, F64 if f64 else torch.float32, 1e-4 if f64 else 1e-1)
        nrhs = case["nrhs"]
        K, y = K.to(F64), y.to(F64)
        x, ld, at = [], [], 0
        mats = torch.split(K, [n * n for n in sizes])
        for m, v in zip(mats, torch.split(y, sizes)):
            n = v.numel()
            a = m.view(n, n)
            L = torch.linalg.cholesky_ex(a)[0]
            x.append(torch.cholesky_solve(v[:, None], L)[:, 0].repeat(nrhs))
            ld.append(2.0 * torch.log(torch.diagonal(L)).sum())
            a.copy_(torch.triu(L.t()) + torch.tril(a, -1))        # column-major lower = row-major upper
        return {"K": K, "x": torch.cat(x), "logdet": torch.stack(ld), "info": None}
    if kind == "gp_batch":
        sizes, K, y = _kernels(case, seed, F64, 1e-4)
        val, dK, dy = [], [], []
        for m, v in zip(torch.split(K, [n * n for n in sizes]), torch.split(y, sizes)):
            r = _gp(m.view(v.numel(), -1), v)
            val.append(r[0])
            dK.append(r[1].reshape(-1))
            dy.append(r[2])
        return {"value": torch.stack(val), "dK": torch.cat(dK), "dy": torch.cat(dy)}
    if kind == "cholesky":
        n = case["n"]
        K = _se_kernel(n, _gen(seed, 5), 1e-2)
        G = _rand((n, n), _gen(seed, 6)).tril_()
        L = torch.linalg.cholesky(K)
        phi = torch.tril(L.t() @ G)
        phi.diagonal().mul_(0.5)
        s = torch.linalg.solve_triangular(L.t(), phi, upper=True)
        s = torch.linalg.solve_triangular(L, s, upper=False, left=False)
        return {"L": L, "dK": 0.5 * (s + s.t())}
    K = _se_kernel(case["n"], _gen(seed, 5), 1e-2)
    v, dK, dy = _gp(K, torch.randn(case["n"], dtype=F64, device="cuda", generator=_gen(seed, 6)))
    return {"value": v, "dK": dK, "dy": dy}


def _gp(K, y):
    """log marginal likelihood of one kernel matrix and its gradients"""
    n = y.numel()
    L = torch.linalg.cholesky_ex(K)[0]
    al = torch.cholesky_solve(y[:, None], L)[:, 0]
    v = -0.5 * (y * al).sum() - torch.log(torch.diagonal(L)).sum() - 0.5 * n * math.log(2 * math.pi)
    return v, 0.5 * (al[:, None] * al[None, :] - torch.cholesky_inverse(L)), -al
