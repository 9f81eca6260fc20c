"""FP64 / complex128 elimination (csrc/inverse.cu) of matrices whose rows have
several scales: the panels' products run on the digit kernels, which keep a row's
and a column's entries relative to its largest."""

import numpy as np
import pytest
import torch

from jaxhps_gb300 import _native as nat

pytestmark = pytest.mark.gpu


def _inverse(A):
    info = torch.zeros(A.shape[0], dtype=torch.int32, device="cuda")
    X = nat.inverse(torch.as_tensor(A, device="cuda"), info=info)
    assert not info.any()
    return X.cpu().numpy()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n,batch", [(140, 3), (193, 160), (257, 2), (600, 1)])
@pytest.mark.parametrize("k,kind", [(0, "big"), (10, "big"), (30, "big"), (60, "big"), (30, "small"), (900, "small"),
                                    (60, "spread")])
def test_rows_of_several_scales(cuda, n, batch, cplx, k, kind):
    """diag(r) A0 has the inverse A0^-1 diag(1 / r).  One row in 16 larger or smaller by
    2^k (a panel's pivot rows are then of two scales), or all of them spread over 2^k:
    no further from it than four times the multiply-adds' own elimination, or than
    n cond(A0) 2^-53 of the largest entry."""
    rng = np.random.default_rng(n + k)
    A0 = rng.standard_normal((n, n)) + 3 * np.sqrt(n) * np.eye(n)
    if cplx:
        A0 = A0 + 1j * rng.standard_normal((n, n))
    some = np.arange(n) % 16 == 3
    r = 2.0 ** (-k * rng.uniform(0, 1, n)) if kind == "spread" else np.where(some, 2.0 ** (k if kind == "big" else -k), 1.0)
    X0 = np.linalg.inv(A0)
    X0 = X0 + X0 @ (np.eye(n) - A0 @ X0)
    A = np.broadcast_to(r[:, None] * A0, (batch, n, n)).copy()
    got = np.abs(_inverse(A) * r - X0).max() / np.abs(X0).max()
    lib = nat.load_library()
    before = lib.hps_gemm_policy(0)
    try:
        chain = np.abs(_inverse(A) * r - X0).max() / np.abs(X0).max()
    finally:
        lib.hps_gemm_policy(before)
    tol = max(4 * chain, n * np.linalg.cond(A0, np.inf) * 2.0 ** -53)
    assert got <= tol, (got, chain, tol)


def test_infinities_and_nan_rows_stay_in_their_matrix(cuda):
    rng = np.random.default_rng(3)
    A = rng.standard_normal((3, 150, 150)) + 40 * np.eye(150)
    A[1, 7, 9], A[1, 20] = np.inf, A[1, 20] * 2.0 ** 40
    info = torch.zeros(3, dtype=torch.int32, device="cuda")
    X = nat.inverse(torch.as_tensor(A, device="cuda"), info=info).cpu().numpy()
    for b in (0, 2):
        assert np.abs(X[b] @ A[b] - np.eye(150)).max() <= 150 * np.linalg.cond(A[b], np.inf) * 2.0 ** -53
