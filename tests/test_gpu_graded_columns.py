"""Refined FP64 / complex128 inverses (csrc/inverse_refined.cu) of matrices whose
columns have several scales, through the leaf stage with an operator that is
any matrix.  The digit products cut a row's entries 2^-62 below its largest:
beyond a span of 2^9 a column would lose bits that no residual shows.  What is
accepted (info = 0) is an FP64 inverse row by row; the rest is handed back."""

import ctypes as C

import numpy as np
import pytest
import torch

from jaxhps_gb300 import _native as nat

pytestmark = pytest.mark.gpu


def _inverses(A, batch, flag):
    """(A^-1 by the leaf stage, status words) of `batch` copies of A."""
    L = nat.lib()
    n, n_cb, ng = A.shape[0], 8, 4
    n_pts, cplx = n + n_cb, np.iscomplexobj(A)
    dt = torch.complex128 if cplx else torch.float64
    # a complex matrix is rows of phases times a real one: coefficients are per point
    phase = np.exp(1j * np.arange(n_pts)) if cplx else np.ones(n_pts)
    op = np.zeros((1, n_pts, n_pts))
    op[0, n_cb:, n_cb:] = (A / phase[n_cb:, None]).real if cplx else A
    op[0, n_cb:, :n_cb] = 1.0
    t = lambda a, d=torch.float64: torch.as_tensor(np.array(a, order="C"), dtype=d, device="cuda")  # noqa: E731
    ops, P, Q = t(op), t(np.ones((n_cb, ng)), dt), t(np.ones((ng, n_pts)), dt)
    co = t(np.broadcast_to(phase, (1, batch, n_pts)), dt)
    Y, T, X = (torch.empty(s, dtype=dt, device="cuda") for s in ((batch, n_pts, ng), (batch, ng, ng), (batch, n, n)))
    info = torch.full((batch,), 9, dtype=torch.int32, device="cuda")
    a = nat.LeafDtnArgs(dtype=nat.TORCH_TO_HPS[dt] | flag, coef_complex=int(cplx), n_leaves=batch, n_pts=n_pts, n_cb=n_cb,
                        n_gauss=ng, nsrc=0, n_ops=1, ops=ops.data_ptr(), coeffs=co.data_ptr(), source=None,
                        P=P.data_ptr(), Q=Q.data_ptr(), Y=Y.data_ptr(), T=T.data_ptr(), v=None, h=None,
                        Aii_inv=X.data_ptr(), info=info.data_ptr(), workspace=None, workspace_bytes=0)
    ws = nat.workspace(L.hps_local_solve_dtn_workspace_size(C.byref(a)), torch.device("cuda"))
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    assert L.hps_local_solve_dtn(C.byref(a), nat.stream_ptr()) == 0
    return X.cpu().numpy(), info.tolist()


def _within(A):
    """Whether every column has an entry within 2^9 of its row's largest (binary orders
    of the larger part; the leaf's scaling of rows leaves them as they are)."""
    e = np.frexp(np.maximum(np.abs(A.real), np.abs(A.imag)))[1].astype(float)
    return (e - e.max(1, keepdims=True)).max(0).min() >= -9


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n,batch", [(65, 1), (96, 3), (200, 80)])
@pytest.mark.parametrize("k", [0, 7, 11, 20, 40])
def test_what_is_accepted_is_inverted(cuda, k, n, batch, cplx):
    """A0 diag(2^-k for every second column) has the inverse diag(2^k) A0^-1, row by
    row: elimination, which does not depend on the columns' scales, and a
    refinement to FP64 are both within n cond(A0) 2^-53 of a row's largest entry.
    Accepted are the matrices within the span (2^-20 and 2^-40 are not).  (200, 80)
    splits its operands ahead of the products, the others do not."""
    rng = np.random.default_rng(n + k)
    A0 = rng.standard_normal((n, n)) + 3 * np.sqrt(n) * np.eye(n)
    if cplx:
        A0 = np.exp(1j * np.arange(8, n + 8))[:, None] * A0
    c = np.where(np.arange(n) % 2, 2.0 ** -k, 1.0)
    X0 = np.linalg.inv(A0)
    X0 = X0 + X0 @ (np.eye(n) - A0 @ X0)
    tol = n * np.linalg.cond(A0, np.inf) * 2.0 ** -53
    X, info = _inverses(A0 * c, batch, nat.HPS_INVERSE_REFINED)
    within = _within(A0 * c)
    assert within or k > 7
    assert set(info) == {0 if within else nat.INFO_NOT_REFINED}
    if not within:
        X, info = _inverses(A0 * c, batch, 0)
        assert set(info) == {0}
    err = np.abs(X * c[:, None] - X0).max(2) / np.abs(X0).max(1)
    assert err.max() <= tol, (err.max(), tol)


def test_the_largest_spans_meet_over_the_rows(cuda):
    """A column is within the span when one row says so, in whichever warp, block
    or half of the columns that row and column are; a column of zeros never is."""
    n = 130
    rng = np.random.default_rng(1)
    A0 = np.eye(n) + 2.0 ** -30 * rng.standard_normal((n, n))
    X, info = _inverses(A0, 5, nat.HPS_INVERSE_REFINED)
    assert set(info) == {0}
    assert np.abs(X @ A0 - np.eye(n)).max() <= n * 2.0 ** -52
    for j in (0, 31, 64, 129):
        A = A0.copy()
        A[:, j] *= 2.0 ** -11
        A[j, (j + 1) % n] = 1.0          # its row keeps its scale
        assert set(_inverses(A, 5, nat.HPS_INVERSE_REFINED)[1]) == {nat.INFO_NOT_REFINED}


@pytest.mark.parametrize("j", [None, 5, 4097])
def test_more_columns_than_a_block_keeps(cuda, j):
    """n = 4100: the columns' spans in two parts.  Accepted and inverted to n 2^-53 times
    the residual's growth (|X| |A| <= 4 for a diagonal of 3 and rows of norm 1 beside
    it), or handed back with one column 2^-20 below the others."""
    n = 4100
    rng = np.random.default_rng(0)
    A = rng.standard_normal((n, n)) / np.sqrt(n) + 3 * np.eye(n)
    if j is not None:
        A[:, j] *= 2.0 ** -20
    X, info = _inverses(A, 1, nat.HPS_INVERSE_REFINED)
    assert info == [0 if j is None else nat.INFO_NOT_REFINED]
    if j is None:
        R = torch.as_tensor(A, device="cuda") @ torch.as_tensor(X[0], device="cuda") - torch.eye(n, device="cuda")
        assert float(R.abs().max()) <= 4 * n * 2.0 ** -53
