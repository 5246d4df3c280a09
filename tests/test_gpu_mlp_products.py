"""The proposal network's BF16 products at the edges of their pipeline: one chunk of K, one more
than the stages of either tile width hold, and the sizes between which the tile width changes.

Tolerance: products of two BF16 numbers are exact in FP32, so an entry is off by at most K
roundings (truncations) of 2^-23 of the sum of its terms' sizes, |A| |B|^T."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from helmholtzbem_gb300 import _capi as C  # noqa: E402


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (128, 256, 512), (256, 128, 576), (384, 128, 1088),
                                   (1920, 1280, 448), (2432, 1024, 384), (2432, 1024, 64),
                                   (256, 2432, 448), (384, 1664, 384), (384, 1664, 64)])
def test_products(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    A = torch.randn((M, K), generator=g).to(torch.bfloat16).cuda()
    B = torch.randn((N, K), generator=g).to(torch.bfloat16).cuda()
    out = torch.full((M, N), float("nan"), device="cuda")
    C.check(C.lib().hbem_bf16_gemm_device(M, N, K, ctypes.c_void_p(A.data_ptr()), K, ctypes.c_void_p(B.data_ptr()), K,
                                          ctypes.c_void_p(out.data_ptr()), N, 1))
    a, b = A.double(), B.double()
    bound = K * 2.0 ** -23 * (a.abs() @ b.abs().T)
    assert bool(((out.double() - a @ b.T).abs() <= bound).all())
    assert np.isfinite(out.sum().item())
