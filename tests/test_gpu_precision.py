"""GPU tests of the accuracy of the factors, against the factor in extended
precision (80-bit on the host).

For a diagonally dominant matrix (entries uniform in [-0.5, 0.5], n added to the
diagonal) the error of the factor is that of its diagonal: every subtraction from
a(i,i) ~ n rounds by at most u n, all else is smaller by a factor of n.  With m
such roundings of variance at most u^2 / 3 (relative, independent), l(i,i) =
sqrt(a(i,i)) has half their error and one rounding of its own, so the factor is
off by at most about u / sqrt(3) sqrt(m / 4 + 1).  The products of a panel of 32
columns are summed by themselves and subtracted once; inside a 32-wide diagonal
block the columns are subtracted one after the other (15.5 on average).  Were
every product rounded at the size of a(i,i), m would be n / 2."""
import ctypes

import numpy as np
import pytest

import dplasma_b200 as db

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def dominant(n, seed, dtype=np.float64):
    g = np.random.default_rng(seed)
    a = g.uniform(-0.5, 0.5, (n, n))
    a = np.tril(a) + np.tril(a, -1).T
    a[np.diag_indices(n)] += n
    return np.ascontiguousarray(a.astype(dtype))


def factor_extended(A):
    A = A.astype(np.longdouble)
    n = A.shape[0]
    L = np.zeros_like(A)
    for j in range(n):
        c = A[j:, j] / np.sqrt(A[j, j])
        L[j:, j] = c
        A[j + 1:, j + 1:] -= np.multiply.outer(c[1:], c[1:])
    return L


def relative_error(F, L):
    return float(np.linalg.norm((F.astype(np.longdouble) - L).astype(np.float64)) / np.linalg.norm(L.astype(np.float64)))


def bound(u, m):
    return u / np.sqrt(3.0) * np.sqrt(m / 4 + 1)


@pytest.mark.parametrize("dtype,u", [(np.float64, 2.0 ** -53), (np.float32, 2.0 ** -24)])
@pytest.mark.parametrize("n,count", [(96, 1400), (96, 400), (200, 700), (300, 290), (512, 3)])   # every shape
def test_batched_factor(gpu_ctx, n, count, dtype, u):
    mats = [dominant(n, s, dtype) for s in range(2)]
    dev = [torch.from_numpy(mats[i % 2].copy()).cuda() for i in range(count)]
    info, _ = gpu_ctx.posv_batched(dev)
    assert int(info.abs().max()) == 0
    for A, F in zip(mats, dev[:2]):
        err = relative_error(np.triu(F.cpu().numpy()).T, factor_extended(A))
        assert err <= bound(u, 15.5 + n / 64), err / u


@pytest.mark.parametrize("n,nb", [(100, 256), (128, 128), (300, 256), (512, 128)])
def test_dense_factor(gpu_ctx, n, nb):
    # 128-wide blocks: 1.5 panels of 32 on average before an entry inside its block,
    # and one subtraction per block column to the left of it
    A = dominant(n, n)
    buf = torch.from_numpy(A.copy()).cuda()
    torch.cuda.synchronize()
    d = db.attach(db.desc_general(n, n, nb, nb, storage=db.STORAGE_LAPACK, lda=n), buf)
    assert gpu_ctx.dpotrf(db.Lower, d) == 0, gpu_ctx.last_error()
    err = relative_error(np.triu(buf.cpu().numpy()).T, factor_extended(A))
    assert err <= bound(2.0 ** -53, 15.5 + 1.5 + n / 256), err * 2.0 ** 53


def growing(n):
    """A = L L^T, exact (all entries dyadic), with L bidiagonal (1 and -1.25) in its
    first 128 columns: the inverse of those grows to 1.25^128 = 3e12, the inverses of
    their 32-wide diagonal blocks to 5 * 1.25^32 = 6e3."""
    g = np.random.default_rng(n)
    L = np.zeros((n, n))
    i = np.arange(128)
    L[i, i] = 1.0
    L[i[1:], i[:-1]] = -1.25
    L[128:, :128] = g.integers(-8, 9, (n - 128, 128)) / 8.0
    L[128:, 128:] = 4.0 * np.eye(n - 128)
    return L @ L.T


@pytest.mark.parametrize("entry,n,nb", [("potrf", 160, 256), ("potrf", 256, 256), ("dtd", 256, 256), ("noalloc", 256, 256),
                                        ("noalloc", 512, 512)])
def test_rows_below_an_ill_conditioned_block(gpu_ctx, entry, n, nb):
    # A solve of the rows below by 32-wide blocks leaves a residual of at most
    # 32 u |D| |L| <= 32 u 2.25 * 6.4e3 times the rows; a product with the inverse of
    # the 128 columns one of about 3e12 u.
    A = growing(n)
    if entry == "potrf":
        d = db.desc_general(n, n, nb, nb, storage=db.STORAGE_LAPACK, lda=n)
    else:
        d = db.desc_sym(n, nb, db.Lower)
    buf = torch.from_numpy(db.pack(np.asfortranarray(A), d)).cuda()
    torch.cuda.synchronize()
    db.attach(d, buf)
    if entry == "noalloc":
        rc = db.lib().dplasma_b200_dpotrf_noalloc(None, db.Lower, ctypes.byref(d))
    else:
        rc = (gpu_ctx.dpotrf if entry == "potrf" else gpu_ctx.dpotrf_dtd)(db.Lower, d)
    assert rc == 0, gpu_ctx.last_error()
    F = np.tril(db.unpack(buf.cpu().numpy(), d)).astype(np.longdouble)
    R = (A[128:, :128] - F[128:, :128] @ F[:128, :128].T).astype(np.float64)
    assert np.linalg.norm(R) <= 32 * 2.0 ** -53 * 2.25 * 6.4e3 * np.linalg.norm(F[128:, :128].astype(np.float64))
