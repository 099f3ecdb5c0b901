"""Device matrices that are 8-byte but not 16-byte aligned (a view into a larger
buffer).  The kernels' bulk and asynchronous copies and tensor maps take 16-byte
addresses, so such a matrix is worked on in a copy, like any storage other than
whole aligned device tiles, and every call gives what it gives for an aligned
one."""
import ctypes

import numpy as np
import pytest

import dplasma_b200 as db


@pytest.mark.parametrize("nb", [128, 256, 512])
@pytest.mark.parametrize("offset,in_place", [(0, 1), (8, 0), (16, 1), (24, 0)])
def test_unaligned_storage_is_copied(nb, offset, in_place):
    d = db.desc_sym(4 * nb, nb, db.Lower)
    d.location = db.DEVICE
    d.mat = 0x7F0000000000 + offset                # never read: the rule looks at the address
    assert db.lib().dplasma_b200_debug_in_place(db.Lower, ctypes.byref(d)) == in_place


def _spd(n):
    g = np.random.default_rng(n)
    a = g.uniform(-0.5, 0.5, (n, n))
    a = np.tril(a) + np.tril(a, -1).T
    a[np.diag_indices(n)] += n
    return np.asfortranarray(a)


def _device(dense, nb, off):
    """descriptor of lower tiles whose storage starts `off` doubles into a buffer"""
    import torch
    n = dense.shape[0]
    d = db.desc_sym(n, nb, db.Lower)
    host = torch.from_numpy(db.pack(dense, d))
    buf = torch.empty(host.numel() + 2, dtype=torch.float64, device="cuda")
    view = buf[off:off + host.numel()]
    view.copy_(host)
    torch.cuda.synchronize()
    assert view.data_ptr() % 16 == 8 * (off % 2)
    return db.attach(d, view), view, buf


def _columns(torch, values, n, nb):
    """device right-hand sides (three columns) and their descriptor"""
    b = values.clone()
    torch.cuda.synchronize()
    return b, db.attach(db.desc_general(n, 3, nb, nb, storage=db.STORAGE_LAPACK, lda=n), b)


@pytest.mark.gpu
@pytest.mark.parametrize("n,nb", [(128, 128), (256, 256), (1024, 256), (1536, 512)])
def test_unaligned_matrix(gpu_ctx, n, nb):
    import torch
    ctx, A = gpu_ctx, _spd(n)
    rhs = torch.from_numpy(np.random.default_rng(1).uniform(-0.5, 0.5, 3 * n)).cuda()
    calls = {
        "potrf": lambda d, b, x: ctx.dpotrf(db.Lower, d),
        "posv": lambda d, b, x: ctx.dposv(db.Lower, d, b),
        "rec": lambda d, b, x: db.lib().dplasma_dpotrf_rec(ctx.h, db.Lower, ctypes.byref(d), nb // 2),
        "dtd": lambda d, b, x: ctx.dpotrf_dtd(db.Lower, d),
        "potrs": lambda d, b, x: ctx.dpotrf(db.Lower, d) or ctx.dpotrs(db.Lower, d, b),
        "trsm": lambda d, b, x: ctx.dtrsm(db.Left, db.Lower, db.Trans, db.NonUnit, 2.0, d, b),
        "potri": lambda d, b, x: ctx.dpotri(db.Lower, d),
        "lansy": lambda d, b, x: 0 if ctx.dlansy(db.InfNorm, db.Lower, d) > n else 1,
    }
    if nb == 256:
        calls["sposv"] = lambda d, b, x: ctx.dsposv(db.Lower, d, b, x)[0]
    for name, call in calls.items():
        out = []
        for off in (0, 1):
            d, view, buf = _device(A, nb, off)
            b, dB = _columns(torch, rhs, n, nb)
            x, dX = _columns(torch, torch.zeros_like(rhs), n, nb)
            assert call(d, dB, dX) == 0, (name, off, ctx.last_error())
            out.append((view.clone(), b, x))
        for p, q in zip(*out):
            if name == "sposv":            # the residual's sums are unordered: rounding after refinement
                assert (p - q).abs().max() <= 1e-13 * p.abs().max(), name
            else:
                assert torch.equal(p, q), name


@pytest.mark.gpu
def test_unaligned_noalloc():
    import torch
    f = db.lib().dplasma_b200_dpotrf_noalloc
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for n, nb in ((128, 128), (512, 512)):
        L = []
        for off in (0, 1):
            d, view, buf = _device(_spd(n), nb, off)
            assert f(stream, db.Lower, ctypes.byref(d)) == 0
            L.append(view.clone())
        assert torch.equal(L[0], L[1])
    d, view, buf = _device(_spd(512), 256, 1)          # two tile rows: refused, nothing is launched
    before = view.clone()
    assert f(stream, db.Lower, ctypes.byref(d)) == db.ERR_NOT_SUPPORTED
    assert torch.equal(view, before)
