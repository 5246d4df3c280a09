"""Small-matrix kernels.  The dense kernel's FP32 stage at the edges of its column layouts: orders below, at and past
a change of the leading dimension or of the columns' register count, and the largest that fits.

T = U diag(s) V^H with s known: sigma_min = 0.1, the others in [0.4, 1].  Tolerances: sigma is
a Ritz value, off by rounding (n eps |T| times a few) and by the square of the vectors' error.
The vectors: the FP32 stage leaves at most n eps32 |T| / gap = 106 * 6e-8 / 0.3 = 2e-5 outside
the near block, which the inverse iterations take down by a factor of 3^-8 = 1.5e-4 at least,
to 3e-9; sigma' = Re u^H T' v with |T'| about 2 is first order in that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import api  # noqa: E402


@pytest.mark.parametrize("nmat", [3, 17])   # a pair of CTAs per matrix, one CTA per matrix
@pytest.mark.parametrize("n", [2, 9, 15, 16, 24, 25, 56, 57, 104])
def test_known_singular_values(n, nmat):
    rng = np.random.default_rng(100 * n + nmat)
    mats, ref = [], []
    for _ in range(nmat):
        z = rng.standard_normal((4, n, n)) + 1j * rng.standard_normal((4, n, n))
        U, V = np.linalg.qr(z[0])[0], np.linalg.qr(z[1])[0]
        s = rng.permutation(np.concatenate([[0.1], np.linspace(0.4, 1.0, n - 1)]))
        T1 = z[2] / np.sqrt(2.0 * n)
        i = int(np.argmin(s))
        mats.append([(U * s) @ V.conj().T, T1])
        ref.append([0.1, (U[:, i].conj() @ T1 @ V[:, i]).real])
    got, ref = np.array(api.sv_dense(mats, d=1)), np.array(ref)
    assert np.abs(got[:, 0] - ref[:, 0]).max() <= 16 * n * np.finfo(float).eps
    assert np.abs(got[:, 1] - ref[:, 1]).max() <= 1e-7


@pytest.mark.parametrize("n", [2, 13, 33, 64, 97])
def test_arnoldi_pairs_of_ctas_give_the_same_bits(n):
    """76 matrices run on pairs of CTAs, 77 on one CTA each."""
    rng = np.random.default_rng(n)
    mats = [[rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))] for _ in range(77)]
    a, b = api.arnoldi_sv(mats[:76], 1, return_status=True), api.arnoldi_sv(mats, 1, return_status=True)
    for x, y in zip(a, b):
        assert np.array_equal(np.asarray(x)[:76], np.asarray(y)[:76], equal_nan=True)


@pytest.mark.parametrize("count", [6, 8, 9, 14])
def test_arnoldi_block_widths(count):
    """Blocks of 12, 16, 18 and 28 columns: the Ritz step's rotations on half-warps up to 16, on
    whole warps beyond.  Ritz values at a relative residual of 1e-9 are off by its square, and
    by rounding: n eps |T|^2 / sigma^2 times a few, 60 * 2.2e-16 * 100 * 4 = 5e-12."""
    n, rng = 60, np.random.default_rng(count)
    s = np.linspace(0.1, 1.0, n)
    mats = []
    for _ in range(3):
        z = rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))
        mats.append([(np.linalg.qr(z[0])[0] * s) @ np.linalg.qr(z[1])[0].conj().T])
    got = api.arnoldi_sv(mats, count, acc=1e-9)[:, :, 0]
    assert np.abs(got / s[:count] - 1).max() <= 5e-12
