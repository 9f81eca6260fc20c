"""The block-structured products of a merge as one grouped launch of the digit
kernel (gemm_groups in csrc/gemm_f64_tc.cu) against the products of the dense
matrices, in which the blocks outside the rectangles are zeros."""

import numpy as np
import pytest
import torch

from jaxhps_gb300 import _stages as st
from jaxhps_gb300._index_maps import oct_merge_maps_dtn, quad_merge_maps_dtn, quad_merge_maps_iti

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,q,nm,scale", [
    ("quad", 2, 3, 1.0), ("quad", 7, 5, 1.0), ("quad", 14, 300, 1.0), ("quad", 33, 2, 1.0), ("quad", 130, 1, 1.0),
    ("oct", 3, 3, 1.0), ("oct", 6, 13, 1.0), ("oct", 8, 2, 1.0), ("oct", 12, 1, 1.0),
    ("iti", 7, 5, 1.0), ("iti", 16, 70, 1.0), ("iti", 33, 2, 1.0), ("quad", 14, 2, np.inf), ("iti", 7, 2, np.nan)])
def test_grouped_products_match_the_dense_ones(cuda, monkeypatch, kind, q, nm, scale):
    """Odd and even blocks (16- and 8-byte aligned), K from 4 to 432, groups
    below and above a tile of 128 x 64; an infinity or a NaN in one child.
    Random children plus a multiple of the identity: D is well conditioned, and
    each product carries at most K 2^-53 of its largest terms on either side,
    2e-13 for K = 1728, and D^-1 is of order 1/8: 1e-12."""
    maps = {"quad": quad_merge_maps_dtn, "oct": lambda n: oct_merge_maps_dtn(n * n), "iti": quad_merge_maps_iti}[kind](q)
    iti = kind == "iti"
    rng = np.random.default_rng(q + nm)
    shape = (nm * maps.nch, maps.nb, maps.nb)
    T = rng.standard_normal(shape) / maps.nb
    if iti:
        T = 0.3 * (T + 1j * rng.standard_normal(shape) / maps.nb)
    else:
        T = T + 4.0 * np.eye(maps.nb)
    if scale != 1.0:
        T[1, 0, 1] = scale
    h = rng.standard_normal((nm * maps.nch, maps.nb, 2)) + (0j if iti else 0.0)
    T, h = torch.as_tensor(T, device=cuda), torch.as_tensor(h, device=cuda)
    out = {}
    for rects in (True, False):
        monkeypatch.setattr(st, "_RECTS", rects)
        r = st.merge_level_dtn(T, h, maps, keep_D_inv=True, keep_BD_inv=True, keep_B=True, iti=iti)
        out[rects] = [x for x in r if isinstance(x, torch.Tensor)]
    assert len(out[True]) == len(out[False]) >= 4
    for a, b in zip(out[True], out[False]):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        if scale != 1.0:
            # what the non-finite child does not reach is the same; it reaches all of its merge
            a, b = a.reshape(nm, -1)[1:], b.reshape(nm, -1)[1:]
        assert np.isfinite(b).all()
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.complex64, torch.complex128])
@pytest.mark.parametrize("ns", [1, 2, 3, 8, 9, 70])
def test_grouped_rows_of_right_hand_sides(cuda, monkeypatch, dtype, ns):
    """h_out += B g~ on the block rows, up to 8 columns on the row kernel and
    above on the products' own: against the dense product, K eps with K = 54
    (n_int) and a factor of 8 for |B| |g~| over |h_out|."""
    iti = dtype.is_complex
    maps = quad_merge_maps_iti(27) if iti else oct_merge_maps_dtn(9)
    rng = np.random.default_rng(ns)
    T = rng.standard_normal((2 * maps.nch, maps.nb, maps.nb)) / maps.nb + (0.0 if iti else 4.0 * np.eye(maps.nb))
    h = rng.standard_normal((2 * maps.nch, maps.nb, ns))
    T, h = (torch.as_tensor(x, device=cuda).to(dtype) for x in (T, h))
    out = []
    for rects in (True, False):
        monkeypatch.setattr(st, "_RECTS", rects)
        out.append([x for x in st.merge_level_dtn(T, h, maps, iti=iti)[:4]])
    eps = torch.finfo(dtype).eps
    for a, b in zip(*out):
        assert float((a - b).abs().max()) <= 8 * maps.n_int * eps * float(b.abs().max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.complex64])
@pytest.mark.parametrize("kind,q,nm", [("2d", 2, 3), ("2d", 7, 300), ("2d", 14, 2), ("2d", 33, 2), ("2d", 64, 1), ("2d", 127, 1),
                                       ("2d", 128, 1), ("3d", 3, 5), ("3d", 5, 2), ("3d", 11, 1)])
def test_grouped_fp32_products_match_the_dense_ones(cuda, monkeypatch, dtype, kind, q, nm):
    """gemm_groups_kernel's three tiles, partial slices of 16 and segments side by
    side, and blocks of 128 that stay with the single products.  The same D^-1
    either way; S and T_out differ by the order of K <= 4 q (3D 12 q^2) terms:
    K eps of the largest entry, 4 for the sums of magnitudes over it."""
    iti = dtype.is_complex
    if iti and kind == "3d":
        pytest.skip("impedance merges are two-dimensional")
    maps = oct_merge_maps_dtn(q * q) if kind == "3d" else quad_merge_maps_iti(q) if iti else quad_merge_maps_dtn(q)
    rng = np.random.default_rng(q)
    shape = (nm * maps.nch, maps.nb, maps.nb)
    T = rng.standard_normal(shape) / maps.nb
    T = 0.3 * (T + 1j * rng.standard_normal(shape) / maps.nb) if iti else T + 4.0 * np.eye(maps.nb)
    T = torch.as_tensor(T, device=cuda).to(dtype)
    out = []
    for rects in (True, False):
        monkeypatch.setattr(st, "_RECTS", rects)
        r = st.merge_level_dtn(T, None, maps, keep_D_inv=True, keep_BD_inv=True, iti=iti)
        out.append((r[0], r[2], r[4], r[5]))
    assert torch.equal(out[0][2], out[1][2])
    eps = torch.finfo(dtype).eps
    for a, b in zip(*out):
        assert float((a - b).abs().max()) <= 4 * maps.n_int * eps * float(b.abs().max())
