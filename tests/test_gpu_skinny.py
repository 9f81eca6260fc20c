"""Products with up to 8 columns, several rows of A to a warp (gemm_skinny_kernel
in csrc/gemm.cu): row counts around the rows of a warp and of a CTA, on both
sides of the rule, K not a multiple of the lanes, odd leading dimensions."""

import pytest
import torch

from jaxhps_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.complex64, torch.complex128])
@pytest.mark.parametrize("M,N,K,batch,pad", [(1, 1, 33, 9000, 0), (3, 1, 32, 4000, 1), (4, 1, 100, 2432, 0), (5, 2, 47, 2000, 0),
                                             (33, 1, 196, 400, 1), (31, 2, 64, 400, 0), (57, 4, 56, 300, 0), (129, 8, 61, 90, 0),
                                             (300, 3, 70, 33, 2), (200, 7, 40, 60, 0), (40, 1, 300, 2, 0)])
def test_products_of_few_columns(cuda, dtype, M, N, K, batch, pad):
    """Against the product in complex128 / FP64: (K + 2) roundings of the sum of
    the magnitudes (complex ones 2 sqrt 2 as large); FP64 against its own sum in
    another order, twice that."""
    g = torch.Generator(device=cuda).manual_seed(M * K + N)

    def draw(*s):
        x = torch.randn(*s[:-1], s[-1] + pad, dtype=torch.float64, device=cuda, generator=g)
        if dtype.is_complex:
            x = torch.complex(x, torch.randn(x.shape, dtype=torch.float64, device=cuda, generator=g))
        return x.to(dtype)[..., : s[-1]]

    A, B, D = draw(batch, M, K), draw(batch, K, N), draw(batch, M, N)
    wide = torch.complex128 if dtype.is_complex else torch.float64
    C = D.to(wide)
    ref = -1.0 * (A.to(wide) @ B.to(wide)) + 2.0 * C
    size = A.abs().double() @ B.abs().double() + 2.0 * C.abs()
    lib = nat.load_library()
    lib.hps_gemm_policy(0)
    try:
        nat.gemm(A, B, D, -1.0, 2.0, Cmat=D)
    finally:
        lib.hps_gemm_policy(1)
    eps = torch.finfo(dtype).eps
    assert bool(((D.to(wide) - ref).abs() <= 2 * (K + 2) * (2 * 2 ** 0.5 if dtype.is_complex else 1) * eps * size).all())
