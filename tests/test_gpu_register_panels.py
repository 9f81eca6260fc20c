"""The panel of the blocked Gauss-Jordan inverse with a row per thread
(gje_panel_reg_kernel in csrc/inverse.cu): every type at the smallest and the
largest n it takes, narrow last panels, partial warps, few and many matrices."""

import numpy as np
import pytest
import torch

from jaxhps_gb300 import _native as nat

pytestmark = pytest.mark.gpu

TYPES = {"f32": (torch.float32, np.float32), "f64": (torch.float64, np.float64),
         "c64": (torch.complex64, np.complex64), "c128": (torch.complex128, np.complex128)}


@pytest.mark.parametrize("kind,n,batch", [
    ("f32", 225, 3), ("f32", 256, 160), ("f32", 481, 1), ("f32", 512, 5), ("f32", 513, 2), ("f64", 65, 2), ("f64", 129, 200),
    ("f64", 255, 1), ("f64", 256, 7), ("f64", 257, 2), ("c64", 129, 1), ("c64", 256, 170), ("c64", 301, 2), ("c64", 512, 3),
    ("c64", 513, 1), ("c128", 65, 1), ("c128", 112, 160), ("c128", 256, 3), ("c128", 258, 1),
    # over a cluster: 2 to 8 CTAs, uneven last CTAs, more than 32 offers, 16 CTAs, and beyond its rows
    ("c64", 257, 4), ("c64", 385, 2), ("c64", 1025, 1), ("f32", 897, 3), ("f32", 2100, 1), ("f64", 700, 2), ("f64", 2049, 1),
    ("c128", 1100, 1), ("c128", 400, 40), ("f32", 4500, 1)])
def test_inverse_with_register_panels(cuda, kind, n, batch):
    """|A X - I| <= 16 n eps |A| |X| in the row-sum norm: the elimination's own
    bound with a growth of 16, for diagonally dominant matrices with their rows
    permuted, so that every pivot has to be looked for."""
    dt, npdt = TYPES[kind]
    rng = np.random.default_rng(n + batch)
    A = rng.standard_normal((batch, n, n))
    if kind[0] == "c":
        A = A + 1j * rng.standard_normal(A.shape)
    A = A + 2 * np.sqrt(n) * np.eye(n)
    A = np.ascontiguousarray(A[:, rng.permutation(n)]).astype(npdt)
    info = torch.full((batch,), 7, dtype=torch.int32, device=cuda)
    X = nat.inverse(torch.as_tensor(A, device=cuda), info=info.zero_()).cpu().numpy()
    assert (info.cpu().numpy() == 0).all()
    wide = np.complex128 if kind[0] == "c" else np.float64
    for b in sorted({0, batch // 2, batch - 1}):
        R = A[b].astype(wide) @ X[b].astype(wide) - np.eye(n)
        S = (np.abs(A[b]).astype(np.float64) @ np.abs(X[b])).sum(1).max()
        assert np.abs(R).sum(1).max() <= 16 * n * np.finfo(npdt).eps * S


@pytest.mark.parametrize("kind,n", [("f32", 300), ("f64", 200), ("c64", 260), ("c128", 130)])
def test_register_panels_report_singular_and_spread_nan(cuda, kind, n):
    dt, npdt = TYPES[kind]
    A = np.stack([np.eye(n)] * 4)[:, ::-1].copy()
    A[1, :, 37] = 0.0            # no pivot in the second panel
    A[2, 5, n - 2] = np.nan
    A[3] = np.eye(n)[::-1] * 2.0 ** np.arange(-30, 30, 60 / n)[:n, None]
    info = torch.zeros(4, dtype=torch.int32, device=cuda)
    X = nat.inverse(torch.as_tensor(A.astype(npdt), device=cuda), info=info).cpu().numpy()
    inf = info.cpu().numpy()
    assert inf[0] == 0 and inf[1] == 38 and inf[3] == 0
    assert np.array_equal(X[0], np.eye(n)[::-1]) and np.isnan(X[2]).any()
    assert np.allclose(X[3] @ A[3], np.eye(n), atol=4 * np.finfo(npdt).eps)


@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 17, 24, 25, 31, 32, 33, 40, 41, 48, 49, 56, 57, 63, 64])
def test_small_fp64_inverse_by_rows(cuda, n):
    """inv_rows_f64_kernel at the edges of its instances, in place, strided, and
    with a zero column and a NaN in one matrix each; bound as above."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((5, n, n + 3)) + 2 * np.sqrt(n) * np.eye(n, n + 3)
    A = np.ascontiguousarray(A[:, rng.permutation(n)])
    A[3, :, n // 2] = 0.0
    A[4, 0, n - 1] = np.nan
    t = torch.as_tensor(A, device=cuda)[..., :n]
    info = torch.zeros(5, dtype=torch.int32, device=cuda)
    X = nat.inverse(t, out=t, info=info).cpu().numpy()
    inf = info.cpu().numpy()
    assert (inf[:3] == 0).all() and inf[3] == n // 2 + 1 and np.isnan(X[4]).any()
    for b in range(3):
        R = A[b, :, :n] @ X[b] - np.eye(n)
        S = (np.abs(A[b, :, :n]) @ np.abs(X[b])).sum(1).max()
        assert np.abs(R).sum(1).max() <= 16 * n * 2.0 ** -52 * S
