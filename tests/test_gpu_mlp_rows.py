"""The proposal network on a batch of more rows than 32 times the 65,535 that a grid's y takes: each
row's output is that of a small batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import api  # noqa: E402


def test_forward_of_two_million_rows():
    net = api.MLP(2, 16, 1, 3, seed=3)
    rows = 32 * 65535 + 1
    X = np.stack([np.linspace(-1, 1, rows), np.linspace(3, 0, rows)], 1).astype(np.float32)
    Y = net.forward(X)
    for part in (slice(0, 100), slice(rows // 2, rows // 2 + 100), slice(rows - 100, rows)):
        assert np.array_equal(Y[part], net.forward(X[part]))
