"""The complex128 trailing update on the tensor cores (exact products of BF16 digits,
zgemm_tc.cu) inside the LU, where it can go wrong: trailing orders at the tiles' edges (128
rows, 32 columns) and their remainders, several matrices, rows and columns of very
different size, integers, a non-finite entry.  ||P A - L U|| stays within the n eps ||L|| ||U||
of an FP64 factorisation and within twice the FMA form's (set_option "lu_tensor_cores" 0): one
rounding per update of depth 32 instead of 64, plus digits cut at 2^-56 of a row's
largest entry."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import _capi as C  # noqa: E402

EPS = 2.220446049250313e-16


def factor(mats, tc):
    import torch
    nm, n = mats.shape[:2]
    F = torch.from_numpy(np.ascontiguousarray(mats.transpose(0, 2, 1))).cuda()
    piv = torch.empty((nm, n), dtype=torch.int32, device="cuda")
    C.check(C.lib().hbem_set_option(b"lu_tensor_cores", tc))
    try:
        C.check(C.lib().hbem_lu_factor_batch_device(n, nm, ctypes.c_void_p(F.data_ptr()), n * n,
                                                    ctypes.c_void_p(piv.data_ptr()), None))
    finally:
        C.check(C.lib().hbem_set_option(b"lu_tensor_cores", 1))
    return F.cpu().numpy().transpose(0, 2, 1), piv.cpu().numpy()


def residual(A, LU, piv):
    n = A.shape[0]
    L, U, P = np.tril(LU, -1) + np.eye(n), np.triu(LU), A.copy()
    for k, p in enumerate(piv):
        P[[k, p]] = P[[p, k]]
    return np.linalg.norm(P - L @ U), n * EPS * np.linalg.norm(L) * np.linalg.norm(U)


def make(kind, nm, n):
    rng = np.random.default_rng(n)
    A = rng.normal(size=(nm, n, n)) + 1j * rng.normal(size=(nm, n, n))
    if kind == "columns":
        A = A * np.logspace(0, -9, n)
    if kind == "rows":
        A = A * rng.permutation(np.logspace(-60, 60, n))[None, :, None]
    if kind == "integers":
        A = rng.integers(-3, 4, (nm, n, n)) + 1j * rng.integers(-3, 4, (nm, n, n))
    if kind == "sparse":
        A[rng.uniform(size=A.shape) < 0.7] = 0
    return np.ascontiguousarray(A, np.complex128)


@pytest.mark.parametrize("kind,nm,n", [("plain", 1, 159), ("plain", 1, 160), ("plain", 3, 161), ("plain", 2, 191),
                                       ("plain", 1, 289), ("plain", 2, 321), ("columns", 1, 300), ("rows", 1, 300),
                                       ("integers", 2, 257), ("sparse", 1, 300)])
def test_lu_residual(kind, nm, n):
    A = make(kind, nm, n)
    (tc, ptc), (fma, pfma) = factor(A, 1), factor(A, 0)
    for m in range(nm):
        r, bound = residual(A[m], tc[m], ptc[m])
        r0, _ = residual(A[m], fma[m], pfma[m])
        assert r <= bound and r <= 2 * r0, (kind, n, r / bound, r / r0)


def test_non_finite_entries_show():
    A = make("plain", 1, 200)
    A[0, 3, 150] = np.nan
    LU, _ = factor(A, 1)
    assert not np.isfinite(LU).all()
