"""FP32 and complex64 products of the TMA + tcgen05 kernel with 128 x 128
tiles (csrc/gemm_tc_wide.cu) at the edges of its tiles, stages and layouts.

Tolerance: 3xTF32 keeps 22 bits of each operand and drops lo x lo, 3 x 2^-22
of |A||B| per product, and the tensor core accumulates in FP32 with
truncation, 2^-23 of the partial sums at each step of 8: together
(3 x 2^-22 + (K / 8 + 2) 2^-23) |A||B| (complex: twice the real steps, |.| of
the parts), and 2^-23 |C| for the addition."""

import numpy as np
import pytest
import torch

from jaxhps_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.fixture
def tensor_cores(cuda):
    lib = nat.load_library()
    lib.hps_gemm_policy(2)
    yield lib
    lib.hps_gemm_policy(1)


def _pair(rng, shape, cplx):
    x = rng.standard_normal(shape).astype(np.float32)
    return (x + 1j * rng.standard_normal(shape).astype(np.float32)).astype(np.complex64) if cplx else x


def _abs(x):
    return np.abs(x.real) + np.abs(x.imag) if np.iscomplexobj(x) else np.abs(x)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("M,N,K,batch,pad", [
    (1, 68, 4, 1, 0), (127, 128, 31, 2, 0), (128, 129, 32, 1, 0), (129, 127, 33, 3, 0), (128, 66, 36, 200, 0),
    (260, 260, 100, 2, 4), (130, 390, 8, 1, 4), (64, 128, 700, 5, 0), (200, 200, 196, 80, 0), (256, 130, 64, 3, 1)])
def test_tile_edges(tensor_cores, M, N, K, batch, pad, cplx):
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    A, B, C = _pair(rng, (batch, M, K + pad), cplx), _pair(rng, (batch, K, N + pad), cplx), _pair(rng, (batch, M, N), cplx)
    dt = torch.complex64 if cplx else torch.float32
    At, Bt, Ct = (torch.as_tensor(t, dtype=dt, device="cuda") for t in (A, B, C))
    a, b = At[..., :K], Bt[..., :N]
    wide = np.complex128 if cplx else np.float64
    for alpha, c, left in ((1.0, None, a), (-1.0, Ct, a), (0.5, Ct, a[0])):
        D = torch.full((batch, M, N + pad), float("nan"), dtype=dt, device="cuda")[..., :N]
        if c is None:
            nat.gemm(left, b, D, alpha)
        else:
            nat.gemm(left, b, D, alpha, 1.0, Cmat=c)
        Ah = (A[..., :K] if left is a else A[:1, :, :K]).astype(wide)
        Bh = B[..., :N].astype(wide)
        ref = alpha * (Ah @ Bh) + (0 if c is None else C)
        steps = (2 * K if cplx else K) / 8 + 2
        tol = (3 * 2.0 ** -22 + steps * 2.0 ** -23) * (_abs(Ah) @ _abs(Bh)) + 2.0 ** -23 * (0 if c is None else _abs(C))
        err = _abs(D.cpu().numpy() - ref)
        assert (err <= tol).all(), float((err / tol).max())
    assert tensor_cores.hps_gemm_tc_status() == 0
