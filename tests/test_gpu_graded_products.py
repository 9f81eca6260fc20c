"""hps_gemm_batched in FP64 and complex128: multiply-adds for any operands, and the
digit kernels (csrc/gemm_f64_tc.cu) where the caller asks for them."""

import numpy as np
import pytest
import torch

from jaxhps_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.fixture
def policy(cuda):
    lib = nat.load_library()
    yield lib.hps_gemm_policy
    lib.hps_gemm_policy(1)


def _draw(rng, shape, cplx):
    x = rng.standard_normal(shape)
    return torch.as_tensor(x + 1j * rng.standard_normal(shape) if cplx else x, device="cuda")


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("M,N,K,batch", [(130, 70, 49, 1), (196, 56, 196, 40), (256, 8, 128, 300), (33, 9, 16, 2)])
@pytest.mark.parametrize("k", [20, 60, 400])
def test_columns_graded_against_rows(cuda, k, M, N, K, batch, cplx):
    """(A 2^-s) (2^s B) = A B for any whole s per step of K: every entry carries what K
    multiply-adds round, K 2^-53 of the sum of the magnitudes (complex: four times)."""
    rng = np.random.default_rng(k + K)
    A, B = _draw(rng, (batch, M, K), cplx), _draw(rng, (batch, K, N), cplx)
    e = rng.integers(0, k + 1, K)
    down, up = (torch.as_tensor(np.ldexp(1.0, x), device="cuda") for x in (-e, e))
    D = torch.empty((batch, M, N), dtype=A.dtype, device="cuda")
    nat.gemm((A * down).contiguous(), (B * up[:, None]).contiguous(), D)
    tol = 2 * (4 if cplx else 1) * K * 2.0 ** -53     # on either side
    assert bool(((D - A @ B).abs() <= tol * (A.abs() @ B.abs())).all())


@pytest.mark.parametrize("cplx", [False, True])
def test_digits_on_request(policy, cplx):
    """The same bits as under the policy that sends every product to the tensor cores;
    without the request, those of the policy that sends none; an unknown flag is refused."""
    rng = np.random.default_rng(2)
    A, B, C = (_draw(rng, s, cplx) for s in ((30, 190, 100), (30, 100, 70), (30, 190, 70)))

    def run(pol, **kw):
        policy(pol)
        D = torch.empty_like(C)
        nat.gemm(A, B, D, -1.0, 1.0, Cmat=C, **kw)
        return D

    assert torch.equal(run(1, digits=True), run(2))
    assert torch.equal(run(1), run(0)) and torch.equal(run(0, digits=True), run(0))
    assert not torch.equal(run(1), run(2))
    lib, dt = nat.load_library(), nat.TORCH_TO_HPS[C.dtype]
    one = (nat.C.c_double * 2)(1.0, 0.0)
    bad = lib.hps_gemm_batched(dt | 0x800, 2, 2, 2, one, A.data_ptr(), 2, 0, B.data_ptr(), 2, 0, one, None, 0, 0,
                               C.data_ptr(), 2, 0, 1, nat.stream_ptr())
    assert bad != 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.complex64])
def test_digits_mean_nothing_in_single_precision(policy, dtype):
    rng = np.random.default_rng(4)
    A, B = _draw(rng, (3, 130, 140), dtype.is_complex).to(dtype), _draw(rng, (3, 140, 130), dtype.is_complex).to(dtype)
    a, b = torch.empty((3, 130, 130), dtype=dtype, device="cuda"), torch.empty((3, 130, 130), dtype=dtype, device="cuda")
    assert torch.equal(nat.gemm(A, B, a), nat.gemm(A, B, b, digits=True))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("N", [1, 2, 4, 8])
def test_few_columns_on_either_kernel(policy, N, cplx):
    """N <= 8 columns on the row-per-warp kernel and on the digit kernel, each asked for:
    both within K 2^-53 of the sum of the magnitudes (complex: four times).  At 608 x
    128 x 512 the rule sends all but real N = 1 (which reads A faster than it is
    converted) to the digits."""
    rng = np.random.default_rng(N)
    A, B = _draw(rng, (608, 128, 512), cplx), _draw(rng, (608, 512, N), cplx)
    out = []
    for pol in (0, 2, 1):
        policy(pol)
        D = torch.empty((608, 128, N), dtype=A.dtype, device="cuda")
        nat.gemm(A, B, D, digits=True)
        out.append(D)
    tol = 2 * (4 if cplx else 1) * 512 * 2.0 ** -53
    assert bool(((out[0] - out[1]).abs() <= tol * (A.abs() @ B.abs())).all())
    assert torch.equal(out[2], out[0 if N == 1 and not cplx else 1])
    assert not torch.equal(out[0], out[1])
