"""A NaN in a matrix is not a zero pivot: the dense, randomized and Arnoldi sigma report it as
values (NaN, or 0 where no column is the largest) and an iteration that does not converge, in the
shared-memory kernels (one CTA and pairs) as behind them; a zero column still is one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import _capi as C, api  # noqa: E402


def mats(n, nmat, value, d=0):
    rng = np.random.default_rng(n)
    M = rng.normal(size=(nmat, d + 1, n, n)) + 1j * rng.normal(size=(nmat, d + 1, n, n))
    M[:, 0, :, n // 2] = value
    return list(M)


@pytest.mark.parametrize("nmat", [1, 20])
@pytest.mark.parametrize("n", [8, 50, 100])
def test_dense_sigma(n, nmat):
    out = api.sv_dense(mats(n, nmat, np.nan, 2), d=2)
    assert np.isnan(out[:, 0]).all()


@pytest.mark.parametrize("n", [20, 100, 130])
def test_randomized_sigma(n):
    R = np.asarray(api.randGaussian(n, 6, seed=1))
    out = api.rsvd_sv(mats(n, 2, np.nan), R, q=1)
    assert not (out > 0).any()
    with pytest.raises(C.HbemError, match="pivot"):
        api.rsvd_sv(mats(n, 2, 0.0), R, q=1)


@pytest.mark.parametrize("n", [20, 100, 130])
@pytest.mark.parametrize("nmat", [1, 100])
def test_arnoldi(n, nmat):
    C.check(C.lib().hbem_set_option(b"arnoldi_maxit", 3))
    try:
        _, status = api.arnoldi_sv(mats(n, nmat, np.nan), count=2, return_status=True)
        _, zero = api.arnoldi_sv(mats(n, nmat, 0.0), count=2, return_status=True)
    finally:
        C.check(C.lib().hbem_set_option(b"arnoldi_maxit", 1000))
    assert (status == 6).all() and (zero == 5).all()
