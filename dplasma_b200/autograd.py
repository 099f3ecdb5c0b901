"""torch.autograd functions over the library's C ABI.

* ``cholesky(A)``: lower Cholesky factor of a symmetric positive definite
  float64 CUDA matrix; forward is ``dplasma_dpotrf``, backward
  ``dplasma_dpotrf_adjoint`` (the reverse Cholesky sweep; the gradient returned
  for A is symmetric).
* ``gp_log_marginal_likelihood_batched(Ks, ys)``: the same for a list of
  independent problems; forward is one batched launch
  (``dplasma_b200_dposv_batched``: factor, solve, log-det), backward one
  (``dplasma_b200_gp_gradient_batched``: the K_i^-1 and the gradients from
  them), with all problems in one flat buffer so that the rest is a fixed
  number of whole-batch tensor operations on vectors; ``se_kernel_batched`` builds the K_i the
  same way, and ``gp_log_marginal_likelihood_flat`` takes the batch as one
  flat tensor (one autograd node).
* ``gp_log_marginal_likelihood(K, y)``: ``-1/2 y^T K^-1 y - 1/2 log det K
  - n/2 log 2 pi`` for a Gaussian-process kernel matrix K and targets y
  (vector or n x m); forward is one factorization and one solve
  (``dplasma_dpotrf`` + ``dplasma_dpotrs``), backward
  ``dK = 1/2 alpha alpha^T - 1/2 K^-1`` with ``K^-1`` -- the Cholesky adjoint
  of the log-determinant (``Lbar = diag(2 / L(i,i))``) -- formed from the
  factor by ``dplasma_b200_gp_gradient``, and ``dy = -alpha``.  Gradients with respect to
  parameters of K (a lengthscale, ...) follow by torch's own chain rule.

Matrices cross the C ABI as LAPACK-storage device descriptors: a row-major
torch tensor is the column-major transpose, so a symmetric K reads the same,
and the column-major lower factor appears as the upper triangle of the
row-major buffer.
"""
from __future__ import annotations

import ctypes
import math

import torch

from . import Context, desc_general, attach, lib, Lower, STORAGE_LAPACK, torch_ready

_ctx = {}


def context(device=None) -> Context:
    d = torch.device("cuda" if device is None else device)
    idx = d.index if d.index is not None else torch.cuda.current_device()
    if idx not in _ctx:
        _ctx[idx] = Context(idx)
    return _ctx[idx]


def _lapack_desc(buf: torch.Tensor, n: int, m: int | None = None, nb: int = 256):
    m = n if m is None else m
    d = desc_general(n, m, nb, nb, storage=STORAGE_LAPACK, lda=max(n, 1))
    attach(d, buf)
    return d


def _check_square(A: torch.Tensor):
    if not (A.is_cuda and A.dtype == torch.float64 and A.dim() == 2 and A.shape[0] == A.shape[1]):
        raise ValueError("expected a square float64 CUDA matrix")


def _factor(A: torch.Tensor):
    """column-major lower factor in a row-major buffer (its upper triangle)"""
    n = A.shape[0]
    buf = A.detach().contiguous().clone()
    torch_ready(buf)
    ctx = context(A.device)
    info = ctx.dpotrf(Lower, _lapack_desc(buf, n))
    if info != 0:
        raise RuntimeError(f"dplasma_dpotrf: INFO = {info} (matrix not positive definite)" if info > 0
                           else f"dplasma_dpotrf: {info} {ctx.last_error()}")
    return buf


def _adjoint(Lrow: torch.Tensor, Lbar: torch.Tensor) -> torch.Tensor:
    """Abar (symmetric) from L and Lbar given as ordinary (row-major, lower) tensors."""
    n = Lrow.shape[0]
    ctx = context(Lrow.device)
    Lc = Lrow.t().contiguous()              # column-major L
    Bc = torch.tril(Lbar).t().contiguous()  # column-major Lbar (lower)
    torch_ready(Lc, Bc)
    rc = ctx.dpotrf_adjoint(Lower, _lapack_desc(Lc, n), _lapack_desc(Bc, n))
    if rc != 0:
        raise RuntimeError(f"dplasma_dpotrf_adjoint: {rc} {ctx.last_error()}")
    up = torch.triu(Bc)                      # column-major lower part = row-major upper
    return up + torch.triu(Bc, 1).t()


def _plain(g: torch.Tensor) -> bool:
    """Whether a kernel may read g and nobody differentiates or batches what
    comes of it (create_graph, is_grads_batched)."""
    if g.requires_grad:
        return False
    try:
        g.data_ptr()
    except RuntimeError:
        return False
    return True


def _gp_gradient(buf: torch.Tensor, rhs: torch.Tensor, g: torch.Tensor) -> torch.Tensor:
    """g / 2 (alpha alpha^T - m K^-1) from the factor as _factor leaves it and
    alpha^T (m x n)."""
    if not _plain(g):
        return g * _gp_gradient(buf, rhs, torch.ones((), dtype=buf.dtype, device=buf.device))
    n = buf.shape[0]
    ctx = context(buf.device)
    # saved tensors come back from a hook with any strides
    buf, rhs, g = buf.contiguous(), rhs.contiguous(), g.contiguous()
    dK = torch.empty_like(buf)
    torch_ready(buf, rhs, g, dK)
    d = _lapack_desc(buf, n)
    rc = lib().dplasma_b200_gp_gradient(ctx.h, ctypes.byref(d), rhs.shape[0], rhs.data_ptr(), g.data_ptr(),
                                        dK.data_ptr())
    if rc != 0:
        raise RuntimeError(f"dplasma_b200_gp_gradient: {rc} {ctx.last_error()}")
    return dK


class _Cholesky(torch.autograd.Function):
    @staticmethod
    def forward(ctx_, A):
        _check_square(A)
        buf = _factor(A)
        L = torch.tril(buf.t())
        ctx_.save_for_backward(L)
        return L

    @staticmethod
    def backward(ctx_, gL):
        (L,) = ctx_.saved_tensors
        return _adjoint(L, gL.contiguous())


def cholesky(A: torch.Tensor) -> torch.Tensor:
    return _Cholesky.apply(A)


class _GPLogML(torch.autograd.Function):
    @staticmethod
    def forward(ctx_, K, y):
        _check_square(K)
        n = K.shape[0]
        Y = y.reshape(n, -1) if y.dim() == 1 else y
        buf = _factor(K)                         # column-major lower factor
        ctx = context(K.device)
        # alpha = K^-1 y by dplasma_dpotrs on the factor (column-major rhs)
        # m x n row-major = n x m column-major; a copy (for one column the
        # transpose is already contiguous and would alias y)
        rhs = Y.detach().t().contiguous().clone()
        torch_ready(rhs)
        rc = ctx.dpotrs(Lower, _lapack_desc(buf, n), _lapack_desc(rhs, n, Y.shape[1]))
        if rc != 0:
            raise RuntimeError(f"dplasma_dpotrs: {rc} {ctx.last_error()}")
        alpha = rhs.t()
        logdet = 2.0 * torch.log(torch.diagonal(buf)).sum()
        m = Y.shape[1]
        val = -0.5 * (Y * alpha).sum() - 0.5 * m * logdet - 0.5 * m * n * math.log(2 * math.pi)
        ctx_.save_for_backward(buf, rhs)
        ctx_.ydim = y.dim()
        return val

    @staticmethod
    def backward(ctx_, g):
        buf, rhs = ctx_.saved_tensors
        # K^-1 (the adjoint of log det K through the factor) and the rank-m term
        dK = _gp_gradient(buf, rhs, g)
        alpha = rhs.t()
        dy = -g * alpha
        if ctx_.ydim == 1:
            dy = dy.reshape(-1)
        return dK, dy


def gp_log_marginal_likelihood(K: torch.Tensor, y: torch.Tensor) -> torch.Tensor:
    return _GPLogML.apply(K, y)


_layouts = {}


class _Layout(dict):
    """A batch's layout; mpad and vpad are made when a padded array is first
    built (64-bit indices of every matrix entry: 0.2 s for 1024 problems)."""

    def __missing__(self, key):
        if key not in ("mpad", "vpad"):
            raise KeyError(key)
        import numpy as np
        nmax, sz = self["nmax"], self["sizes"]
        mpad = np.empty(sum(n * n for n in sz), np.int64)
        vpad = np.empty(sum(sz), np.int64)
        for b, (n, mo, vo) in enumerate(zip(sz, self["moff_h"], self["voff_h"])):
            r = np.arange(n, dtype=np.int64)
            mpad[mo:mo + n * n] = b * nmax * nmax + (r[:, None] * nmax + r[None, :]).ravel()
            vpad[vo:vo + n] = b * nmax + r
        dev = self["moff"].device
        self["mpad"], self["vpad"] = torch.from_numpy(mpad).to(dev), torch.from_numpy(vpad).to(dev)
        return self[key]


def _batch_layout(sizes, device):
    """Flat and padded index maps of a batch of orders `sizes` (cached): every
    problem's matrix lives row-major at moff[b] in one flat buffer and at
    [b, :n, :n] of a (batch, nmax, nmax) padded array; mpad / vpad give the
    padded position of each flat matrix / vector entry."""
    key = (tuple(sizes), str(device))
    lay = _layouts.get(key)
    if lay is not None:
        return lay
    import numpy as np
    sz = np.asarray(sizes, dtype=np.int64)
    B, nmax = len(sz), int(sz.max())
    moff = np.concatenate([[0], np.cumsum(sz * sz)[:-1]]).astype(np.int64)
    voff = np.concatenate([[0], np.cumsum(sz)[:-1]]).astype(np.int64)

    def dev(a):
        return torch.from_numpy(a).to(device)

    lay = _Layout({"B": B, "nmax": nmax, "sizes": list(int(v) for v in sz), "n32": dev(sz.astype(np.int32)),
           "moff": dev(moff), "voff": dev(voff),
           "pid": dev(np.repeat(np.arange(B, dtype=np.int64), sz)), "nf": dev(sz.astype(np.float64)),
           "moff_h": moff.tolist(), "voff_h": voff.tolist()})
    if len(_layouts) > 8:
        _layouts.clear()
    _layouts[key] = lay
    return lay


def _split(flat, offs, sizes, square):
    return [flat[o:o + n * n].view(n, n) if square else flat[o:o + n] for o, n in zip(offs, sizes)]


def _gp_flat_forward(Kflat, y0, lay):
    """values of the batch and (factors, alpha) for the backward; Kflat is
    consumed (overwritten by the factors)"""
    dev = Kflat.device
    ctx = context(dev)
    nb = lay["B"]
    alpha = y0.clone()
    ptrK = Kflat.data_ptr() + 8 * lay["moff"]
    ptrY = alpha.data_ptr() + 8 * lay["voff"]
    logdet = torch.empty(nb, dtype=torch.float64, device=dev)
    info = torch.empty(nb, dtype=torch.int32, device=dev)
    torch_ready(Kflat, alpha, ptrK, ptrY, lay["n32"])
    rc = ctx.posv_batched_arrays(torch.float64, nb, lay["n32"], lay["n32"], ptrK, ptrY, 1, logdet, info)
    if rc != 0:
        raise RuntimeError(f"dplasma_b200_dposv_batched: {rc} {ctx.last_error()}")
    bad = info != 0
    if bool(bad.any()):
        raise RuntimeError(f"batched factorization: INFO {info[bad][:4].tolist()} (not positive definite)")
    dots = torch.zeros(nb, dtype=torch.float64, device=dev).index_add_(0, lay["pid"], y0 * alpha)
    vals = -0.5 * dots - 0.5 * logdet - 0.5 * lay["nf"] * math.log(2 * math.pi)
    return vals, alpha


def _gp_flat_backward(Lflat, alpha, g, lay):
    """(dK flat, dy flat) of the batch from the factors and alpha"""
    dev = Lflat.device
    ctx = context(dev)
    B = lay["B"]
    if not _plain(g):
        dK, _ = _gp_flat_backward(Lflat, alpha, torch.ones(B, dtype=Lflat.dtype, device=dev), lay)
        n2 = lay["n32"].long() ** 2
        return (g.index_select(0, torch.repeat_interleave(torch.arange(B, device=dev), n2)) * dK,
                -g.index_select(0, lay["pid"]) * alpha)
    Lflat, alpha, g = Lflat.contiguous(), alpha.contiguous(), g.contiguous()
    dK = torch.empty_like(Lflat)
    pL = Lflat.data_ptr() + 8 * lay["moff"]
    pal = alpha.data_ptr() + 8 * lay["voff"]
    pdK = dK.data_ptr() + 8 * lay["moff"]
    info = torch.empty(B, dtype=torch.int32, device=dev)
    torch_ready(Lflat, alpha, g, pL, pal, pdK, lay["n32"])
    n32 = lay["n32"].data_ptr()
    rc = lib().dplasma_b200_gp_gradient_batched(ctx.h, B, n32, n32, pL.data_ptr(), pal.data_ptr(), g.data_ptr(),
                                                pdK.data_ptr(), info.data_ptr())
    if rc != 0 or bool((info != 0).any()):
        raise RuntimeError(f"batched inverse failed: {rc} {ctx.last_error()}")
    return dK, -g.index_select(0, lay["pid"]) * alpha


class _GPLogMLBatched(torch.autograd.Function):
    """List form: the problems are gathered into one flat buffer, then one
    batched factor + solve + log-det launch forward and one batched gradient
    launch backward, with a fixed number of whole-batch tensor operations
    around them."""

    @staticmethod
    def forward(ctx_, nb, *args):
        Ks, ys = args[:nb], args[nb:]
        lay = _batch_layout([K.shape[0] for K in Ks], Ks[0].device)
        Kflat = torch.cat([K.detach().reshape(-1) for K in Ks])
        y0 = torch.cat([y.detach().reshape(-1) for y in ys])
        vals, alpha = _gp_flat_forward(Kflat, y0, lay)
        ctx_.lay = lay
        ctx_.yshapes = [y.shape for y in ys]
        ctx_.save_for_backward(Kflat, alpha)
        return vals

    @staticmethod
    def backward(ctx_, g):
        Lflat, alpha = ctx_.saved_tensors
        lay = ctx_.lay
        dKflat, dyflat = _gp_flat_backward(Lflat, alpha, g, lay)
        dKs = _split(dKflat, lay["moff_h"], lay["sizes"], True)
        dys = [v.reshape(sh) for v, sh in zip(_split(dyflat, lay["voff_h"], lay["sizes"], False), ctx_.yshapes)]
        return (None, *dKs, *dys)


class _GPLogMLFlat(torch.autograd.Function):
    """Flat form: Kflat holds the row-major K_i one after the other, yflat
    the y_i; one autograd node for the whole batch."""

    @staticmethod
    def forward(ctx_, Kflat, yflat, sizes):
        lay = _batch_layout(list(sizes), Kflat.device)
        work = Kflat.detach().clone()
        vals, alpha = _gp_flat_forward(work, yflat.detach().contiguous(), lay)
        ctx_.lay = lay
        ctx_.save_for_backward(work, alpha)
        return vals

    @staticmethod
    def backward(ctx_, g):
        Lflat, alpha = ctx_.saved_tensors
        dKflat, dyflat = _gp_flat_backward(Lflat, alpha, g, ctx_.lay)
        return dKflat, dyflat, None


def gp_log_marginal_likelihood_batched(Ks, ys) -> torch.Tensor:
    """Values (batch,) of the GP log-marginal likelihoods of independent
    problems K_i (n_i x n_i, float64 CUDA) and y_i (n_i,)."""
    return _GPLogMLBatched.apply(len(Ks), *Ks, *ys)


def gp_log_marginal_likelihood_flat(Kflat: torch.Tensor, yflat: torch.Tensor, sizes) -> torch.Tensor:
    """The same with the problems concatenated: Kflat the row-major K_i one
    after the other (sum n_i^2 values), yflat the y_i (sum n_i values), sizes
    the n_i.  One autograd node for the batch (use with se_kernel_batched(...,
    flat=True))."""
    return _GPLogMLFlat.apply(Kflat, yflat, tuple(int(n) for n in sizes))


def se_kernel_batched(xs, lengthscale: torch.Tensor, nugget: float = 1e-4, flat: bool = False):
    """se_kernel for a list of point sets x_i (n_i x d) with one shared
    lengthscale, built in a fixed number of whole-batch operations on a
    padded array; returns the K_i as views into one flat tensor, or with
    flat=True that tensor itself (row-major K_i one after the other)."""
    dev = xs[0].device
    lay = _batch_layout([x.shape[0] for x in xs], dev)
    B, nmax, d = lay["B"], lay["nmax"], xs[0].shape[1]
    X = torch.zeros(B * nmax, d, dtype=xs[0].dtype, device=dev).index_copy(0, lay["vpad"], torch.cat(xs, 0))
    X = X.view(B, nmax, d)
    d2 = ((X[:, :, None, :] - X[:, None, :, :]) ** 2).sum(-1)
    Kp = torch.exp(-d2 / (2.0 * lengthscale ** 2)) + nugget * torch.eye(nmax, dtype=X.dtype, device=dev)
    Kflat = Kp.reshape(-1).index_select(0, lay["mpad"])
    return Kflat if flat else _split(Kflat, lay["moff_h"], lay["sizes"], True)


def se_kernel(x: torch.Tensor, lengthscale: torch.Tensor, nugget: float = 1e-4) -> torch.Tensor:
    """Squared-exponential kernel exp(-|xi - xj|^2 / (2 l^2)) + nugget I (torch ops)."""
    d2 = ((x[:, None, :] - x[None, :, :]) ** 2).sum(-1)
    return torch.exp(-d2 / (2.0 * lengthscale ** 2)) + nugget * torch.eye(x.shape[0], dtype=x.dtype, device=x.device)
