"""GPU tests of the launch shapes that follow from sizes: the block order and
the shared-memory POTRF of the FP64 factorization at block and 32-column
edges, re-tiled caller layouts, the one-block-per-CTA sweeps and their column
groups, the batched kernel's warps per problem, and the Gaussian-process
gradients.  Each is compared with numpy / torch in 64 bits; tolerances are
the reference's residual ratio (< 10 in units of N eps) or stated beside."""
import ctypes

import numpy as np
import pytest

import dplasma_b200 as db

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def spd(n, seed, scale=1.0):
    g = np.random.default_rng(seed)
    a = g.uniform(-0.5, 0.5, (n, n))
    a = np.tril(a) + np.tril(a, -1).T
    a[np.diag_indices(n)] += n
    return np.asfortranarray(a * scale)


def dev_desc(dense, nb, uplo, lapack=False):
    n = dense.shape[0]
    d = db.desc_general(n, n, nb, nb, storage=db.STORAGE_LAPACK, lda=n) if lapack else db.desc_sym(n, nb, uplo)
    buf = torch.from_numpy(db.pack(dense, d)).cuda()
    torch.cuda.synchronize()
    return db.attach(d, buf), buf


def factor_ratio(L, A):
    return np.abs(L @ L.T - A).sum(1).max() / (np.abs(A).sum(1).max() * A.shape[0] * EPS)


@pytest.mark.parametrize("n,nb,uplo,lapack", [
    (1, 1, "L", False), (31, 32, "L", False), (33, 128, "U", True), (127, 128, "L", True), (129, 93, "U", False),
    (256, 200, "L", False),            # as many tiles of 128 as of 200: still two layouts
    (257, 256, "L", True), (640, 128, "L", False), (1000, 320, "U", True), (1536, 512, "L", False),
    (6400, 128, "L", False),           # 50 blocks: four panels per update task
    (7937, 256, "L", True)])           # 63 blocks, the last one a single row: six panels
def test_factor_shapes(gpu_ctx, n, nb, uplo, lapack):
    A = spd(n, n)
    up = db.Lower if uplo == "L" else db.Upper
    d, buf = dev_desc(A, nb, up, lapack)
    before = db.unpack(buf.cpu().numpy(), d)
    assert gpu_ctx.dpotrf(up, d) == 0, gpu_ctx.last_error()
    out = db.unpack(buf.cpu().numpy(), d)
    L = np.tril(out) if uplo == "L" else np.triu(out).T
    assert factor_ratio(L, A) < 10.0
    # the other triangle of what is stored is not touched
    other = np.triu if uplo == "L" else np.tril
    assert np.array_equal(other(out, 1 if uplo == "L" else -1), other(before, 1 if uplo == "L" else -1))


@pytest.mark.parametrize("panels", [1, 3, 6, 12, 15])
def test_factor_panels_per_update(panels, monkeypatch):
    # the counts that large orders take, and others, on one of 18 blocks (the last chunk
    # of a column is open)
    monkeypatch.setenv("DPLASMA_B200_F64_CHUNK", str(panels))
    A = spd(2200, panels)
    with db.Context(0) as ctx:
        d, buf = dev_desc(A, 256, db.Lower, True)
        assert ctx.dpotrf(db.Lower, d) == 0, ctx.last_error()
    assert factor_ratio(np.tril(db.unpack(buf.cpu().numpy(), d)), A) < 10.0


@pytest.mark.parametrize("scale", [2.0 ** -990, 2.0 ** 990])
def test_factor_pivots_outside_the_fast_range(gpu_ctx, scale):
    # powers of two: the factor is the scaled factor, to a last place of the
    # root (both roots of a pivot are correct to that)
    n = 300
    A = spd(n, 7)
    d, buf = dev_desc(A * scale, 256, db.Lower, True)
    assert gpu_ctx.dpotrf(db.Lower, d) == 0, gpu_ctx.last_error()
    L = np.tril(db.unpack(buf.cpu().numpy(), d)) / np.sqrt(scale)
    assert factor_ratio(L, A) < 10.0


@pytest.mark.parametrize("n,bad", [(300, 0), (300, 31), (300, 32), (300, 127), (300, 128), (300, 299), (1000, 700)])
@pytest.mark.parametrize("value", [-1.0, 0.0, np.nan])
def test_info_at_block_edges(gpu_ctx, n, bad, value):
    A = spd(n, n)
    A[bad, bad] = value if bad == 0 else A[bad, bad] * 0 + value
    if bad > 0:
        A[bad, :bad] = A[:bad, bad] = 0.0          # the pivot is A(bad, bad) itself
    d, buf = dev_desc(A, 96, db.Lower, True)
    assert gpu_ctx.dpotrf(db.Lower, d) == bad + 1


@pytest.mark.parametrize("n,nrhs", [(100, 1), (200, 9), (300, 33), (385, 16), (512, 64), (700, 40), (2000, 24)])
@pytest.mark.parametrize("uplo", ["L", "U"])
def test_sweep_shapes(gpu_ctx, n, nrhs, uplo):
    g = np.random.default_rng(n + nrhs)
    up = db.Lower if uplo == "L" else db.Upper
    A = spd(n, n)
    d, buf = dev_desc(A, 256, up, True)
    B = g.uniform(-0.5, 0.5, (n, nrhs))
    bB = torch.from_numpy(np.ascontiguousarray(B.T).reshape(-1)).cuda()
    torch.cuda.synchronize()
    dB = db.attach(db.desc_general(n, nrhs, 256, 256, storage=db.STORAGE_LAPACK, lda=n), bB)
    assert gpu_ctx.dposv(up, d, dB) == 0, gpu_ctx.last_error()
    X = bB.cpu().numpy().reshape(nrhs, n).T
    r = np.abs(A @ X - B).sum(1).max()
    assert r / ((np.abs(A).sum(1).max() * np.abs(X).sum(1).max() + np.abs(B).sum(1).max()) * n * EPS) < 10.0


def test_sweep_trace_is_of_the_sweep_that_runs(tmp_path, monkeypatch):
    # one block per CTA: the traced sweep is the chain, and gives the untraced results
    n, nrhs = 4096, 8
    A = spd(n, n)
    B = np.random.default_rng(2).uniform(-0.5, 0.5, (nrhs, n))
    out = []
    for path in ("", str(tmp_path / "wave")):
        monkeypatch.setenv("DPLASMA_B200_WAVE_TRACE", path)
        with db.Context(0) as ctx:
            d, buf = dev_desc(A, 256, db.Lower, True)
            b = torch.from_numpy(B.copy()).cuda()
            torch.cuda.synchronize()
            e = db.attach(db.desc_general(n, nrhs, 256, 256, storage=db.STORAGE_LAPACK, lda=n), b)
            assert ctx.dposv(db.Lower, d, e) == 0, ctx.last_error()
            out.append(b)
    assert torch.equal(out[0], out[1])
    lines = (tmp_path / "wave").read_text().splitlines()
    assert [l.split()[:4] for l in lines] == [["sweep", "chain", "trans", "0"], ["sweep", "chain", "trans", "1"]]
    for l in lines:
        steps = [int(v) for v in l.split("steps_ns")[1].split()]
        assert len(steps) == 8 and all(0 < s < 1000000 for s in steps)


def test_sweep_exchange_buffer_is_bounded():
    # many columns go through the sweep in turns: the workspace is the padded
    # right-hand sides and a bounded exchange buffer, not a second copy of them;
    # the columns repeat, so every turn gives the first one's results
    n, nrhs, period = 512, 49152, 64
    A = spd(n, n)
    with db.Context(0) as ctx:
        d, buf = dev_desc(A, 256, db.Lower, True)
        assert ctx.dpotrf(db.Lower, d) == 0, ctx.last_error()
        b = torch.rand(period, n, dtype=torch.float64, device="cuda").sub_(0.5)
        B = b.repeat(nrhs // period, 1).contiguous()
        torch.cuda.synchronize()

        def solve(cols, t):
            e = db.attach(db.desc_general(n, cols, 256, 256, storage=db.STORAGE_LAPACK, lda=n), t)
            assert ctx.dpotrs(db.Lower, d, e) == 0, ctx.last_error()

        solve(period, b)
        free = torch.cuda.mem_get_info()[0]
        solve(nrhs, B)
        grown = free - torch.cuda.mem_get_info()[0]
    assert grown < 1.5 * 8 * n * nrhs, grown
    X, first = B.view(-1, period, n), b.cpu().numpy()
    assert bool((X == X[0]).all())
    r = np.abs(A @ first.T - A @ X[0].cpu().numpy().T).max()
    assert r <= n * EPS * np.abs(A).sum(1).max() * np.abs(first).max()


def test_sweep_passes_nans_on(gpu_ctx):
    # every NaN payload travels through the sweep's exchange buffer, the one
    # that marks an empty word included
    n, nrhs = 700, 3
    A = spd(n, 1)
    d, buf = dev_desc(A, 256, db.Lower, True)
    B = np.zeros((nrhs, n))
    B[0, 5] = np.nan
    B.view(np.uint64)[1, 300] = 0xFFFFFFFFFFFFFFFF
    bB = torch.from_numpy(B.reshape(-1)).cuda()
    torch.cuda.synchronize()
    dB = db.attach(db.desc_general(n, nrhs, 256, 256, storage=db.STORAGE_LAPACK, lda=n), bB)
    assert gpu_ctx.dposv(db.Lower, d, dB) == 0, gpu_ctx.last_error()
    X = bB.cpu().numpy().reshape(nrhs, n)
    assert np.isnan(X[0]).all() and np.isnan(X[1]).all() and (X[2] == 0).all()


@pytest.mark.parametrize("count,lo,hi,dtype,nrhs,shape", [
    (1200, 90, 96, "f64", 1, "1 warp"), (1300, 80, 96, "f32", 3, "1 warp"), (700, 1, 96, "f64", 1, "4 warps"),
    (700, 90, 96, "f32", 3, "4 warps"), (600, 97, 256, "f64", 2, "8 warps"), (600, 97, 256, "f32", 16, "two per SM"),
    (320, 257, 300, "f64", 1, "8 warps"), (320, 257, 300, "f32", 1, "two per SM"), (3, 500, 512, "f64", 1, "8 warps"),
    (3, 1000, 1024, "f32", 1, "8 warps"), (40, 1, 70, "f64", 4, "8 warps")])
def test_batched_shapes(gpu_ctx, count, lo, hi, dtype, nrhs, shape):
    # kernels with nugget 1: condition <= n + 1, so solutions agree to about n eps times that
    dt = torch.float64 if dtype == "f64" else torch.float32
    g = torch.Generator().manual_seed(count + hi)
    sizes = torch.randint(lo, hi + 1, (count,), generator=g).tolist()
    sizes[0], sizes[-1] = hi, lo
    Ks, ys = [], []
    for n in sizes:
        x = torch.rand(n, 3, generator=g, dtype=torch.float64)
        Ks.append((torch.exp(-12.5 * torch.cdist(x, x) ** 2) + torch.eye(n, dtype=torch.float64)).to(dt).double())
        ys.append(torch.randn(nrhs, n, generator=g, dtype=torch.float64).to(dt).double())
    mats = [K.to(dt).cuda() for K in Ks]
    rhs = [y.to(dt).cuda() for y in ys]
    info, logdet = gpu_ctx.posv_batched(mats, rhs)
    assert (info == 0).all()
    assert shape in gpu_ctx.batched_variant()          # every kernel of bt_variants is among these
    u = EPS if dtype == "f64" else 2.0 ** -24
    for n, K, y, m, r, ld in zip(sizes, Ks, ys, mats, rhs, logdet):
        L = torch.linalg.cholesky(K)
        F = torch.triu(m.double().cpu()).t()
        assert (F - L).norm() <= 10 * n * u * L.norm()
        X = torch.cholesky_solve(y.t(), L).t()
        assert (r.double().cpu() - X).norm() <= 10 * n * (n + 1) * u * X.norm()
        assert abs(ld - 2 * torch.log(torch.diagonal(L)).sum()) <= 10 * n * n * u


@pytest.mark.parametrize("n,scale", [(70, 2.0 ** -990), (300, 2.0 ** 990)])
def test_batched_pivots_outside_the_fast_range(gpu_ctx, n, scale):
    A = spd(n, 3)
    m = torch.from_numpy(np.ascontiguousarray(A * scale)).cuda()
    info, _ = gpu_ctx.posv_batched([m])
    assert int(info[0]) == 0
    assert factor_ratio(np.triu(m.cpu().numpy()).T / np.sqrt(scale), A) < 10.0


@pytest.mark.parametrize("n,m", [(1, 1), (127, 1), (129, 2), (700, 1), (1500, 3), (1, 4), (130, 4), (130, 16),
                                 (255, 17), (300, 700)])
def test_gp_gradient(n, m):
    from dplasma_b200 import autograd as dag
    g = torch.Generator().manual_seed(n)
    x = torch.rand(n, 3, generator=g, dtype=torch.float64)
    K = torch.exp(-12.5 * torch.cdist(x, x) ** 2) + torch.eye(n, dtype=torch.float64)
    y = torch.randn(n, m, generator=g, dtype=torch.float64)
    Kd, yd = K.cuda().requires_grad_(True), y.cuda().requires_grad_(True)
    v = dag.gp_log_marginal_likelihood(Kd, yd)
    dK, dy = torch.autograd.grad(3.0 * v, (Kd, yd))
    Ki = torch.linalg.inv(K)
    al = Ki @ y
    ref = 1.5 * (al @ al.t() - m * Ki)
    tol = 100 * n * (n + 1) * EPS           # condition <= n + 1 (nugget 1)
    assert (dK.cpu() - ref).norm() <= tol * ref.norm() and (dy.cpu() + 3.0 * al).norm() <= tol * al.norm() * 3
    assert torch.equal(dK, dK.t())


def test_gp_gradients_differentiate_and_batch_over_the_outer_gradient():
    # the gradients are linear in the incoming one for whoever differentiates
    # (create_graph) or batches it (is_grads_batched) as for the plain kernel call
    from dplasma_b200 import autograd as dag
    g = torch.Generator().manual_seed(5)
    Ks, ys = [], []
    for n in (65, 40):
        x = torch.rand(n, 3, generator=g, dtype=torch.float64)
        Ks.append((torch.exp(-12.5 * torch.cdist(x, x) ** 2) + torch.eye(n, dtype=torch.float64)).cuda())
        ys.append(torch.randn(n, generator=g, dtype=torch.float64).cuda())
    flat = torch.cat([K.reshape(-1) for K in Ks])
    cases = [(lambda K: dag.gp_log_marginal_likelihood(K, ys[0]), Ks[0]),
             (lambda K: dag.gp_log_marginal_likelihood_flat(K, torch.cat(ys), (65, 40)), flat)]
    for f, K in cases:
        K = K.clone().requires_grad_(True)
        v = f(K)
        w = torch.full_like(v, 2.0).requires_grad_(True)
        (dK,) = torch.autograd.grad(v, K, w, create_graph=True)
        (one,) = torch.autograd.grad(f(K), K, torch.ones_like(v))
        assert torch.allclose(dK, 2.0 * one, rtol=1e-12, atol=1e-12)
        (dw,) = torch.autograd.grad(dK.sum(), w)
        assert torch.allclose(dw.sum(), one.sum(), rtol=1e-9)
        ws = torch.stack([torch.ones_like(v), torch.full_like(v, 3.0)])
        (both,) = torch.autograd.grad(f(K), K, ws, is_grads_batched=True)
        assert torch.allclose(both, torch.stack([one, 3.0 * one]), rtol=1e-12, atol=1e-12)


def test_gp_gradients_through_saved_tensor_hooks():
    # a hook may give the saved factor and solution back with other strides
    from dplasma_b200 import autograd as dag
    g = torch.Generator().manual_seed(6)
    Ks, ys = [], []
    for n in (70, 33):
        x = torch.rand(n, 3, generator=g, dtype=torch.float64)
        Ks.append((torch.exp(-12.5 * torch.cdist(x, x) ** 2) + torch.eye(n, dtype=torch.float64)).cuda())
        ys.append(torch.randn(n, generator=g, dtype=torch.float64).cuda())
    y2 = torch.stack([ys[0], 2 * ys[0] + 1], 1)
    cases = [(dag.gp_log_marginal_likelihood, (Ks[0], ys[0])), (dag.gp_log_marginal_likelihood, (Ks[0], y2)),
             (lambda K, y: dag.gp_log_marginal_likelihood_flat(K, y, (70, 33)).sum(),
              (torch.cat([K.reshape(-1) for K in Ks]), torch.cat(ys))),
             (lambda *t: dag.gp_log_marginal_likelihood_batched(t[:2], t[2:]).sum(), (*Ks, *ys))]

    def spread(t):
        # the same values, no two of them side by side
        return torch.stack([t, torch.full_like(t, 7.0)], -1)[..., 0]

    for f, args in cases:
        args = [a.clone().requires_grad_(True) for a in args]
        plain = torch.autograd.grad(f(*args), args)
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, spread):
            v = f(*args)
        for a, b in zip(torch.autograd.grad(v, args), plain):
            assert torch.equal(a, b)


def test_gp_without_targets():
    # no columns: value and gradient are zero
    from dplasma_b200 import autograd as dag
    n = 200
    K = (torch.eye(n, dtype=torch.float64) * 2.0).cuda().requires_grad_(True)
    y = torch.empty(n, 0, dtype=torch.float64, device="cuda", requires_grad=True)
    v = dag.gp_log_marginal_likelihood(K, y)
    dK, dy = torch.autograd.grad(v, (K, y))
    assert float(v.detach()) == 0.0 and dy.shape == (n, 0) and bool((dK == 0).all())


def test_gp_gradient_refuses(gpu_ctx):
    d = db.desc_general(8, 8, 256, 256, storage=db.STORAGE_LAPACK, lda=8)
    buf = torch.eye(8, dtype=torch.float64, device="cuda")
    db.attach(d, buf)
    f = db.lib().dplasma_b200_gp_gradient
    assert f(None, ctypes.byref(d), 1, None, None, None) == db.ERR_NOT_INITIALIZED
    assert f(gpu_ctx.h, ctypes.byref(d), 1, None, None, None) == db.ERR_ILLEGAL_VALUE
    g, out = torch.ones((), dtype=torch.float64, device="cuda"), torch.empty_like(buf)
    torch.cuda.synchronize()
    assert f(gpu_ctx.h, ctypes.byref(d), 1, None, g.data_ptr(), out.data_ptr()) == db.ERR_ILLEGAL_VALUE
    assert f(gpu_ctx.h, ctypes.byref(d), 0, None, None, out.data_ptr()) == db.ERR_ILLEGAL_VALUE
