"""The randomized sigma of a matrix of any size: scaled by powers of ten up to 1e+-100 (whose squares of
squares leave the range of FP64), it is the unscaled one's times the scale, behind the shared-memory
kernel (orders 110 and above).  Scaling rounds the entries and the sketch's products anew: n eps times
the condition of the smallest singular value's estimate, 1e-10 as for the other matrices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import api  # noqa: E402


@pytest.mark.parametrize("n,s", [(110, 8), (150, 16), (260, 12)])
@pytest.mark.parametrize("scale", [1e-100, 1e-80, 1e80, 1e100])
def test_scaled_matrices(n, s, scale):
    rng = np.random.default_rng(n)
    A = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    R = np.asarray(api.randGaussian(n, s, seed=5))
    one = api.rsvd_sv([[A]], R, q=2)[0, 0]
    got = api.rsvd_sv([[A * scale]], R, q=2)[0, 0] / scale
    assert abs(got - one) <= 1e-10 * one
