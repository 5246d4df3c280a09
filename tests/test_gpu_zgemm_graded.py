"""The complex128 LU's tensor-core update (zgemm_tc.cu) on matrices whose rows and columns are of
different size, entry by entry: |P A - L U| against |L| |U|, where a norm over the matrix shows
its largest rows alone.  Orders with one tile to a CTA and with five and a remainder (the two
buffers, read-ahead and exponents' rounds).

Bound per entry: an update's fixed-point error is at most 2^-38 of its sum |l||u| (64 products of
operands below 2^1 of their exponents, rounded to 2^-56 of it, exponents at most 9 above those of an
entry pair they meet in: 2^(6 + 1 + 2 - 56 + 9)), the rest of an FP64 factorisation's at most
3 n eps, and as much for the residual's own product.  Per row, the residual's norm against |L| |U|'s
is within twice the FMA form's (set_option "lu_tensor_cores" 0): the roundings average alike."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import _capi as C  # noqa: E402

EPS = 2.220446049250313e-16


def make(kind, nm, n):
    rng = np.random.default_rng(n + nm)
    A = rng.normal(size=(nm, n, n)) + 1j * rng.normal(size=(nm, n, n))
    if kind == "rows":
        A *= rng.permutation(np.logspace(-60, 60, n))[None, :, None]
    if kind == "half_rows":
        A *= np.where(rng.permutation(n) < n // 2, 1e-8, 1.0)[None, :, None]
    if kind == "columns":
        A *= rng.permutation(np.logspace(-40, 40, n))
    if kind == "both":
        A *= rng.permutation(np.logspace(-30, 30, n))[None, :, None] * rng.permutation(np.logspace(-30, 30, n))
    if kind == "sparse_rows":
        A[rng.uniform(size=A.shape) < 0.7] = 0
        A *= rng.permutation(np.logspace(-15, 15, n))[None, :, None]
    if kind == "blocks":       # four kinds of entries of very different size, as the blocks of a T(k)
        h = n // 2
        A[:, :h, h:] *= 1e-9
        A[:, h:, :h] *= 1e9
        A[:, h:, h:] *= 1e-3
    if kind == "crossed":      # rows that are large where the others are small: no scaling evens them out
        A *= np.where(np.add.outer(np.arange(n), np.arange(n)) % 3 == 0, 1.0, 1e-10)
    if kind == "far":          # products below 2^-970 that fill whole entries
        A[:, -40:, :] *= 2.0 ** -490
        A[:, :, 100:160] *= 2.0 ** -500
    return np.ascontiguousarray(A, np.complex128)


KINDS = ["plain", "rows", "half_rows", "columns", "both", "sparse_rows", "blocks", "crossed", "far"]


def factor(A, tc):
    import torch
    nm, n = A.shape[:2]
    LU = torch.from_numpy(np.ascontiguousarray(A.transpose(0, 2, 1))).cuda()
    piv = torch.empty((nm, n), dtype=torch.int32, device="cuda")
    C.check(C.lib().hbem_set_option(b"lu_tensor_cores", tc))
    try:
        C.check(C.lib().hbem_lu_factor_batch_device(n, nm, ctypes.c_void_p(LU.data_ptr()), n * n,
                                                    ctypes.c_void_p(piv.data_ptr()), None))
    finally:
        C.check(C.lib().hbem_set_option(b"lu_tensor_cores", 1))
    return LU.transpose(-1, -2), piv.cpu().numpy()


def residual(A, F, piv):
    """|P A - L U| and |L| |U|, rows and columns brought to the size of one (exactly)."""
    import torch
    P = A.copy()
    for k, p in enumerate(piv):
        P[[k, p]] = P[[p, k]]
    L, U = torch.tril(F, -1) + torch.eye(len(A), dtype=torch.complex128, device="cuda"), torch.triu(F)
    r = torch.exp2(-torch.floor(torch.log2(torch.from_numpy(np.abs(P).max(1)).cuda())))[:, None]
    c = torch.exp2(-torch.floor(torch.log2(U.abs().amax(0))))
    L, U, P = r * L, U * c, r * torch.from_numpy(P).cuda() * c
    return (P - L @ U).abs(), L.abs() @ U.abs()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nm,n", [(1, 300), (1, 1200), (3, 700)])
def test_every_entry_of_the_factorisation(kind, nm, n):
    A = make(kind, nm, n)
    (tc, ptc), (fma, pfma) = factor(A, 1), factor(A, 0)
    for m in range(nm):
        res, mag = residual(A[m], tc[m], ptc[m])
        res0, mag0 = residual(A[m], fma[m], pfma[m])
        assert bool((res <= (2.0 ** -38 + 6 * n * EPS) * mag).all()), (kind, m, (res / mag).nan_to_num().max().item())
        rows, rows0 = (res.norm(dim=1) / mag.norm(dim=1)).max().item(), (res0.norm(dim=1) / mag0.norm(dim=1)).max().item()
        assert rows <= 2 * rows0, (kind, m, rows, rows0)


def test_tiles_of_non_finite_columns():
    import torch
    n = 1200
    A = make("plain", 1, n)[0]
    A[700, 1100] = np.nan
    LU = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    C.check(C.lib().hbem_lu_factor_batch_device(n, 1, ctypes.c_void_p(LU.data_ptr()), n * n,
                                                ctypes.c_void_p(piv.data_ptr()), None))
    LU = LU.T.cpu().numpy()
    assert np.isfinite(LU[:, :1100]).all() and not np.isfinite(LU[:, 1100]).all()
