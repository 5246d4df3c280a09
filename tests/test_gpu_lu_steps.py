"""Solves by launches per 32-row block (few columns: k_solve_step with the inverses of the
diagonal blocks), the cluster QR behind the randomized and Arnoldi sigma, where they can go
wrong: orders below, at and above the line (128), remainders of the blocks, one column and
the column pairs' remainder, several matrices.  Residuals of both solve forms against
n eps ||T|| ||X|| (a backward-stable solve's bound has a modest constant: 16 here), and the
randomized sigma against numpy's with the same sketch at 1e-10."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import _capi as C, api  # noqa: E402
from oracle import oracle as O  # noqa: E402


@pytest.mark.parametrize("n", [127, 128, 129, 160, 191, 257, 400])
@pytest.mark.parametrize("nmat,nrhs", [(1, 1), (1, 13), (3, 5), (2, 33)])
def test_solves_leave_small_residuals(n, nmat, nrhs):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + 7 * nrhs)
    A = torch.randn((nmat, n, n), dtype=torch.complex128, device="cuda", generator=g)
    X = torch.randn((nmat, nrhs, n), dtype=torch.complex128, device="cuda", generator=g)
    LU, piv = A.clone(), torch.empty((nmat, n), dtype=torch.int32, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())   # noqa: E731
    C.check(C.lib().hbem_lu_factor_batch_device(n, nmat, p(LU), n * n, p(piv), None))
    for trans in (0, 1):
        Y = X.clone()
        C.check(C.lib().hbem_lu_solve_batch_device(n, nmat, trans, p(LU), n * n, p(piv), nrhs, p(Y), nrhs * n))
        M = A.transpose(-1, -2).cpu().numpy()
        Yh, Xh = Y.transpose(-1, -2).cpu().numpy(), X.transpose(-1, -2).cpu().numpy()
        for m in range(nmat):
            T = M[m] if trans == 0 else M[m].conj().T
            res = np.linalg.norm(T @ Yh[m] - Xh[m], axis=0)
            assert (res <= 16 * n * 2.2e-16 * np.linalg.norm(T, 2) * np.linalg.norm(Yh[m], axis=0)).all()


@pytest.mark.parametrize("n,s", [(255, 12), (256, 12), (300, 1), (301, 17), (270, 32)])
def test_randomized_sigma_matches_numpy(n, s):
    rng = np.random.default_rng(n)
    U, V = (np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))[0] for _ in range(2))
    Ts = [[(U * np.geomspace(1.0, 1e-3, n)) @ V.conj().T], [(V * np.linspace(2.0, 0.1, n)) @ U]]
    R = np.asarray(api.randGaussian(n, s, seed=5))
    got = api.rsvd_sv(Ts, R, q=2)
    for g, (T,) in zip(got[:, 0], Ts):
        ref = O.rsvd_sv(T, R, q=2)
        assert abs(g - ref) <= 1e-10 * ref
