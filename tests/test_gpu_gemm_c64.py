"""Complex64 products in 128 x 64 tiles (gemm_c64_kernel in csrc/gemm.cu): edges
of the tiles and of the K slices of 8, odd leading dimensions (8-byte aligned
rows), C and D the same, sizes on both sides of the rule."""

import numpy as np
import pytest
import torch

from jaxhps_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,batch,pad,alpha,beta", [
    (128, 64, 8, 152, 0, 1.0, 0.0), (127, 63, 7, 160, 0, -1.0, 1.0), (129, 65, 9, 80, 1, 0.5, 2.0), (256, 256, 32, 20, 0, 1.0, 1.0),
    (256, 254, 1, 20, 1, 1.0, 1.0), (100, 33, 33, 160, 3, 1.0 - 0.5j, 0.25j), (65, 65, 16, 200, 0, 1.0, 1.0),
    (64, 64, 16, 200, 0, 1.0, 1.0), (65, 33, 20, 200, 1, 1.0, 1.0), (1000, 700, 31, 2, 0, -1.0, 1.0), (300, 300, 0, 16, 0, 1.0, 2.0)])
def test_products_at_tile_edges(cuda, M, N, K, batch, pad, alpha, beta):
    """Against complex128: (K + 2) roundings of at most 2 sqrt(2) 2^-24 of the
    sum of the magnitudes."""
    g = torch.Generator(device=cuda).manual_seed(M + N + K)

    def draw(*s):
        x = torch.randn(*s[:-1], s[-1] + pad, 2, device=cuda, generator=g)
        return torch.view_as_complex(x)[..., : s[-1]]

    A, B, D = draw(batch, M, K), draw(batch, K, N), draw(batch, M, N)
    wide = torch.complex128
    C = D.to(wide)
    ref = alpha * (A.to(wide) @ B.to(wide)) + beta * C
    size = abs(alpha) * (A.abs().double() @ B.abs().double()) + abs(beta) * C.abs()
    nat.gemm(A, B, D, alpha, beta, Cmat=D)
    assert bool(((D.to(wide) - ref).abs() <= (K + 2) * 2 * 2 ** 0.5 * 2.0 ** -24 * size).all())
