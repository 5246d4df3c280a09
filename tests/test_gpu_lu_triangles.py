"""Solves with factors whose 32 x 32 diagonal blocks are ill-conditioned: discretised smooth kernels
(numerically rank-deficient blocks of U), triangular matrices that grow by products of their
entries, a Vandermonde matrix.  Substitution leaves residuals of a modest constant times
n eps ||T|| ||x|| (16 here, as for the other solves) however ill-conditioned its triangles are; the
launch-per-block form has to as well.  Orders with several blocks and remainders, one column and the
column pairs, several matrices, both directions."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import _capi as C  # noqa: E402


def make(kind, n):
    rng = np.random.default_rng(n)
    t = np.sort(rng.random(n))
    g = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    return {
        "gauss": lambda: np.exp(-10. * np.subtract.outer(t, t) ** 2) + 1e-10 * np.eye(n),
        "hilbert": lambda: 1. / (np.add.outer(np.arange(n), np.arange(n)) + 1.),
        "upper": lambda: np.eye(n) - np.triu(np.ones((n, n)), 1),
        "lower": lambda: np.eye(n) - np.tril(np.ones((n, n)), -1),
        "random_upper": lambda: np.triu(g),
        "vandermonde": lambda: np.vander(np.cos(np.pi * (np.arange(n) + .5) / n)),
        "moderate": lambda: np.eye(n) + .3 * np.triu(g, 1),     # blocks between the well- and the ill-conditioned
    }[kind]().astype(np.complex128)


KINDS = ["gauss", "hilbert", "upper", "lower", "random_upper", "vandermonde", "moderate"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,nmat,nrhs", [(128, 1, 1), (257, 2, 33), (300, 1, 7)])
def test_residuals_as_small_as_substitutions(kind, n, nmat, nrhs):
    import torch
    M = make(kind, n)
    rng = np.random.default_rng(1)
    A = torch.from_numpy(np.ascontiguousarray(np.repeat(M.T[None], nmat, 0))).cuda()
    piv = torch.empty((nmat, n), dtype=torch.int32, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())   # noqa: E731
    C.check(C.lib().hbem_lu_factor_batch_device(n, nmat, p(A), n * n, p(piv), None))
    x = rng.normal(size=(nmat, n, nrhs)) + 1j * rng.normal(size=(nmat, n, nrhs))
    for trans in (0, 1):
        T = M if trans == 0 else M.conj().T
        B = T @ x
        X = torch.from_numpy(np.ascontiguousarray(B.transpose(0, 2, 1))).cuda()
        C.check(C.lib().hbem_lu_solve_batch_device(n, nmat, trans, p(A), n * n, p(piv), nrhs, p(X), nrhs * n))
        Y = X.cpu().numpy().transpose(0, 2, 1)
        res = np.linalg.norm(T @ Y - B, axis=1)
        bound = 16 * n * 2.2e-16 * np.linalg.norm(T, 2) * np.linalg.norm(Y, axis=1)
        assert (res <= bound).all(), (kind, trans, (res / bound).max())
