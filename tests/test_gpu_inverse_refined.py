"""FP64 / complex128 inverses refined from the single-precision inverse
(csrc/inverse_refined.cu) through the leaf and merge stages: what they give
against the elimination, and the way back to it where they do not converge."""

import numpy as np
import pytest
import torch

import jaxhps_gb300 as hps
from jaxhps_gb300 import _native as nat
from jaxhps_gb300 import _stages as st

pytestmark = pytest.mark.gpu


def _pde(p, q, L, c=1.0, iti=False, d=2):
    box = (-1.0, 1.0) * d
    root = hps.DiscretizationNode2D(*box) if d == 2 else hps.DiscretizationNode3D(*box)
    dom = hps.Domain(p=p, q=q, root=root, L=L)
    x = dom.interior_points
    ones = np.ones(x.shape[:2])
    kw = dict(D_xx_coefficients=1 + 0.3 * np.cos(x[..., 0]) ** 2, D_yy_coefficients=ones,
              I_coefficients=c * (1 + 0.2 * np.exp(-(x ** 2).sum(-1))) if np.isscalar(c) else c)
    if d == 3:
        kw["D_zz_coefficients"] = ones
    if iti:
        kw.update(use_ItI=True, eta=4.0)
    return hps.PDEProblem(dom, source=np.sin(x[..., 0]) + x[..., 1], **kw)


def _stages(pde, refined, monkeypatch):
    """(Y, T, v, h, S_lst, g_lst) with the inverses refined or eliminated."""
    from jaxhps_gb300 import _iti, _stages_3D as st3

    if not refined:
        monkeypatch.setattr(st, "refines", lambda dtype, n: False)
    if pde.use_ItI:
        Y, T, v, h = st.local_solve_stage_uniform_2D_ItI(pde)
        out = _iti.merge_stage_uniform_2D_ItI(T, h, l=pde.domain.L)
    elif pde.domain.bool_2D:
        Y, T, v, h = st.local_solve_stage_uniform_2D_DtN(pde)
        out = st.merge_stage_uniform_2D_DtN(T, h, l=pde.domain.L)
    else:
        Y, T, v, h = st.local_solve_stage_uniform_3D_DtN(pde)
        out = st3.merge_stage_uniform_3D_DtN(T, h, l=pde.domain.L)
    monkeypatch.undo()
    return [Y, T, v, h, *out[0], *out[1]]


@pytest.mark.parametrize("p,q,L,iti,d", [(10, 8, 1, False, 2), (11, 9, 2, False, 2), (16, 14, 3, False, 2),
                                         (18, 16, 1, False, 2), (9, 7, 2, True, 2), (16, 14, 2, True, 2),
                                         (7, 5, 1, False, 3), (10, 8, 1, False, 3)])
def test_stages_agree_with_the_elimination(cuda, monkeypatch, p, q, L, iti, d):
    """n = 64 is eliminated either way, 65 to 768 and odd sizes are not.  Both
    are FP64 inverses of matrices with condition numbers of up to about 1e3
    (ItI 1e4): they agree to 1e-11 of the largest entry, as the FP64 stages
    agree with the oracle."""
    pde = _pde(p, q, L, 1.5, iti, d)
    ref = _stages(pde, False, monkeypatch)
    got = _stages(pde, True, monkeypatch)
    for a, b in zip(got, ref):
        assert float((a - b).abs().max()) <= 1e-11 * float(b.abs().max())


def _resonant(p, q):
    """A one-leaf-deep problem whose first leaf is nearly singular: its zero-order
    coefficient is an eigenvalue of the leaf's collocation matrix up to 1e-10."""
    pde = _pde(p, q, 1)
    n_cb = pde.P.shape[0]
    x = pde.domain.interior_points
    A = ((1 + 0.3 * np.cos(x[0, :, 0]) ** 2)[:, None] * pde.D_xx + pde.D_yy)[n_cb:, n_cb:]
    lam = np.linalg.eigvals(A)
    lam = float(-np.real(lam[np.argmin(np.abs(lam))]))
    c = np.ones(x.shape[:2])
    c[0] = lam * (1 + 1e-10)
    return _pde(p, q, 1, c)


def test_a_leaf_that_is_not_refined_is_eliminated(cuda, monkeypatch):
    pde = _resonant(12, 10)
    seen = []
    real = st.unrefined
    monkeypatch.setattr(st, "unrefined", lambda infos: seen.append(real(infos)) or seen[-1])
    Y, T, v, h = st.local_solve_stage_uniform_2D_DtN(pde)
    assert seen == [True]
    monkeypatch.undo()
    ref = _stages(pde, False, monkeypatch)
    for a, b in zip((Y, T, v, h), ref):
        assert torch.equal(a, b)          # the second run is the elimination, bit for bit


@pytest.mark.parametrize("refined", [True, False])
def test_status_words_of_the_c_entry(cuda, refined):
    """-2 for the resonant leaf only, and nothing of it without the flag."""
    import ctypes as C

    pde = _resonant(12, 10)
    L = nat.lib()
    n_cb, ng = pde.P.shape
    n_pts, nl = pde.Q.shape[1], 4
    n_i = n_pts - n_cb
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    cs, ops = pde.active_coefficients()
    ops_t, co, P, Q = t(np.stack(ops)), t(np.stack(cs)), t(pde.P), t(pde.Q)
    Y, T, Ai = (torch.empty(s, dtype=torch.float64, device="cuda")
                for s in ((nl, n_pts, ng), (nl, ng, ng), (nl, n_i, n_i)))
    info = torch.full((nl,), 9, dtype=torch.int32, device="cuda")
    a = nat.LeafDtnArgs(dtype=nat.HPS_F64 | (nat.HPS_INVERSE_REFINED if refined else 0), coef_complex=0, n_leaves=nl,
                        n_pts=n_pts, n_cb=n_cb, n_gauss=ng, nsrc=0, n_ops=len(ops), ops=ops_t.data_ptr(),
                        coeffs=co.data_ptr(), source=None, P=P.data_ptr(), Q=Q.data_ptr(), Y=Y.data_ptr(),
                        T=T.data_ptr(), v=None, h=None, Aii_inv=Ai.data_ptr(), info=info.data_ptr(), workspace=None,
                        workspace_bytes=0)
    ws = nat.workspace(L.hps_local_solve_dtn_workspace_size(C.byref(a)), torch.device("cuda"))
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    assert L.hps_local_solve_dtn(C.byref(a), nat.stream_ptr()) == 0
    assert info.tolist() == ([-2, 0, 0, 0] if refined else [0, 0, 0, 0])
    a.dtype |= 0x200                      # an unknown flag is an unknown type
    assert L.hps_local_solve_dtn(C.byref(a), nat.stream_ptr()) != 0


@pytest.mark.parametrize("p,q,L,iti,d", [(16, 14, 4, False, 2), (17, 15, 4, False, 2), (12, 10, 1, False, 3),
                                         (13, 11, 3, True, 2), (14, 12, 2, True, 2)])
def test_products_of_split_operands(cuda, monkeypatch, p, q, L, iti, d):
    """Stages whose inverses have their operands split ahead of the products
    (rows of at least 192 numbers, 1 GFLOP a product): n = 196, 225, 1000 with a
    merge of 1200, complex 169 and 196.  The bound is that of
    test_stages_agree_with_the_elimination; a leaf with a NaN is handed back
    and leaves the others alone."""
    pde = _pde(p, q, L, 1.5, iti, d)
    ref = _stages(pde, False, monkeypatch)
    got = _stages(pde, True, monkeypatch)
    for a, b in zip(got, ref):
        assert float((a - b).abs().max()) <= 1e-11 * float(b.abs().max())
    if iti or d == 3:
        return
    c = 1.5 * (1 + 0.2 * np.exp(-(pde.domain.interior_points ** 2).sum(-1)))
    c[3, 4 * p - 4 + 40] = np.nan   # an interior point: the equation is not set at the boundary ones
    Y = st.local_solve_stage_uniform_2D_DtN(_pde(p, q, L, c))[0]
    assert bool(torch.isnan(Y[3]).any())
    keep = [i for i in range(Y.shape[0]) if i != 3]
    assert float((Y[keep] - ref[0][keep]).abs().max()) <= 1e-11 * float(ref[0].abs().max())
