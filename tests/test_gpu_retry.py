"""What is run again where an inverse is not refined to FP64: the leaves that were
not, and the merge levels from the first such one on."""

import numpy as np
import pytest
import torch

import jaxhps_gb300 as hps
from jaxhps_gb300 import _native as nat
from jaxhps_gb300 import _stages as st
from jaxhps_gb300._index_maps import quad_merge_maps_dtn

pytestmark = pytest.mark.gpu


# ---------------------------------------------------------------------------
# leaves
# ---------------------------------------------------------------------------


def _leaf_pde(iti, which):
    """256 leaves of 121 points; on those of `which` the zero-order coefficient is an
    eigenvalue of the leaf's collocation matrix up to 1e-10 (DtN)."""
    p = 11
    dom = hps.Domain(p=p, q=9, root=hps.DiscretizationNode2D(-1.0, 1.0, -1.0, 1.0), L=4)
    x = dom.interior_points
    ones = np.ones(x.shape[:2])
    c = ones.copy()
    kw = dict(D_xx_coefficients=ones, D_yy_coefficients=ones)
    if iti:
        kw.update(use_ItI=True, eta=4.0)
    pde = hps.PDEProblem(dom, source=np.sin(x[..., 0]) + x[..., 1], I_coefficients=c, **kw)
    if not iti:
        n_cb = pde.P.shape[0]
        lam = np.linalg.eigvals((pde.D_xx + pde.D_yy)[n_cb:, n_cb:])
        c[which] = float(-np.real(lam[np.argmin(np.abs(lam))])) * (1 + 1e-10)
        pde = hps.PDEProblem(dom, source=np.sin(x[..., 0]) + x[..., 1], I_coefficients=c, **kw)
    return pde


def test_only_the_leaves_that_are_not_refined_are_eliminated(cuda, monkeypatch):
    """Those have the elimination's results (of the same leaves on their own: bit for
    bit), the others what the first run gave them."""
    which = [3, 77, 255]
    pde = _leaf_pde(False, which)
    calls = []
    args = nat.LeafDtnArgs
    monkeypatch.setattr(nat, "LeafDtnArgs", lambda **kw: calls.append((kw["n_leaves"], kw["dtype"])) or args(**kw))
    got = st.local_solve_stage_uniform_2D_DtN(pde, keep_inverse=True)
    assert [n for n, _ in calls] == [256, 3]
    assert [bool(d & nat.HPS_INVERSE_REFINED) for _, d in calls] == [True, False]
    assert not pde._leaf_info.any()
    monkeypatch.setattr(st, "unrefined", lambda infos: False)
    first = st.local_solve_stage_uniform_2D_DtN(pde, keep_inverse=True)
    monkeypatch.undo()
    monkeypatch.setattr(st, "refines", lambda dtype, n: False)
    whole = st.local_solve_stage_uniform_2D_DtN(pde, keep_inverse=True)
    rest = [i for i in range(256) if i not in which]
    for a, b, c in zip(got, first, whole):
        assert torch.equal(a[rest], b[rest])
        assert torch.equal(a[which], c[which])


@pytest.mark.parametrize("iti", [False, True])
@pytest.mark.parametrize("bad", [[0], [5, 9, 200], list(range(0, 256, 2)), list(range(256))])
def test_leaves_handed_back(cuda, monkeypatch, iti, bad):
    """Any leaves marked as not refined: up to half of them are run again alone, the
    result is that of leaves that are all refined, to the 1e-11 between both."""
    pde = _leaf_pde(iti, [])
    leaf = st.local_solve_stage_uniform_2D_ItI if iti else st.local_solve_stage_uniform_2D_DtN
    ref = leaf(pde)
    name = "hps_local_solve_iti" if iti else "hps_local_solve_dtn"
    lib = nat.lib()

    class Marks:
        def __getattr__(self, n):
            return getattr(lib, n)

    marks = Marks()
    seen = []

    def run(a, stream):
        s = getattr(lib, name)(a, stream)
        seen.append(a._obj)
        return s

    setattr(marks, name, run)
    real = st.unrefined

    def mark(infos):
        if len(seen) == 1:
            infos[0][bad] = nat.INFO_NOT_REFINED
        return real(infos)

    monkeypatch.setattr(nat, "lib", lambda: marks)
    monkeypatch.setattr(st, "unrefined", mark)
    got = leaf(pde)
    monkeypatch.undo()
    assert [a.n_leaves for a in seen] == [256, len(bad) if 2 * len(bad) <= 256 else 256]
    assert not pde._leaf_info.any()
    for a, b in zip(got, ref):
        assert float((a - b).abs().max()) <= 1e-11 * float(b.abs().max())


# ---------------------------------------------------------------------------
# merges
# ---------------------------------------------------------------------------


def _record(monkeypatch):
    calls = []
    real = st.merge_level_dtn

    def level(T, h, maps, **kw):
        calls.append((maps.nb, kw.get("refined") is not None))
        return real(T, h, maps, **kw)

    monkeypatch.setattr(st, "merge_level_dtn", level)
    return calls, real


def _children(q, levels, fail, which):
    """DtN-like children (symmetric) of a quadtree whose merge `which` of level `fail`
    has an interface matrix with an eigenvalue of 1e-9, all others of order 1."""
    rng = np.random.default_rng(q + fail)
    n, nb = 4 ** levels, 4 * q
    R = rng.standard_normal((n, nb, nb)) / (4 * nb)
    T = R + R.transpose(0, 2, 1) + 4 * np.eye(nb)
    maps, cur, where = [], torch.as_tensor(T, device="cuda"), None
    for lvl in range(fail):
        maps.append(quad_merge_maps_dtn(q * 2 ** lvl))
        cur = st.merge_level_dtn(cur, None, maps[-1])[2]
    m = quad_merge_maps_dtn(q * 2 ** fail)
    Tc = cur.cpu().numpy()[4 * which:4 * which + 4]
    D = np.zeros((m.n_int, m.n_int))
    for c in range(4):
        at = np.nonzero(m.loc[c] >= 0)[0]
        D[np.ix_(at, at)] += Tc[c][np.ix_(m.loc[c, at], m.loc[c, at])]
    lam = np.linalg.eigvalsh(D)[0] - 1e-9
    for i in range(m.n_int):
        for c, l in zip(m.int_c[i], m.int_l[i]):
            node, at = 4 * which + int(c), int(l)
            for mm in reversed(maps):       # the leaf point that this boundary point is
                node, at = 4 * node + int(mm.ext_c[at]), int(mm.ext_l[at])
            T[node, at, at] -= lam / 2
    return T, rng.standard_normal((n, nb, 2))


@pytest.mark.parametrize("fail,which", [(0, 5), (1, 2), (2, 0)])
def test_levels_below_a_near_singular_merge_stay_refined(cuda, monkeypatch, fail, which):
    """Level by level, refined where that succeeds and eliminated where not: the same
    bits as the stage, which looks at the status words once and goes back."""
    q, levels = 20, 3
    T, h = (torch.as_tensor(a, device="cuda") for a in _children(q, levels, fail, which))
    want, failed, Tl, hl = [], [], T, h
    for lvl in range(levels):
        maps = quad_merge_maps_dtn(q * 2 ** lvl)
        for refined in ([], None):
            out = st.merge_level_dtn(Tl, hl, maps, refined=refined)
            if not st.unrefined(refined):
                break
            failed.append(lvl)
        want.append(out)
        Tl, hl = out[2], out[3]
    assert fail in failed and min(failed) == fail
    calls, _ = _record(monkeypatch)
    S, g, Ttop = st.merge_stage_uniform_2D_DtN(T, h, l=levels, return_T=True)
    monkeypatch.undo()
    for lvl in range(levels):
        assert torch.equal(S[lvl], want[lvl][0]) and torch.equal(g[lvl], want[lvl][1])
    assert torch.equal(Ttop, want[-1][2][0])
    expect = [True] * levels + [True] * fail + [False]
    for lvl in range(fail + 1, levels):
        expect += [True, False] if lvl in failed else [True]
    assert [r for _, r in calls] == expect


def _stage(kind):
    rng = np.random.default_rng(7)
    if kind == "adaptive":
        root = hps.DiscretizationNode2D(0.0, 1.0, 0.0, 1.0)

        def f(x):                      # a ridge along the children's interface: many panels there
            xp = torch if isinstance(x, torch.Tensor) else np
            return xp.exp(-(x[..., 0] - 0.5) ** 2 / 1e-4)

        dom = hps.Domain.from_adaptive_discretization(p=12, q=10, root=root, f=f, tol=1e-6)
        x = dom.interior_points
        pde = hps.PDEProblem(dom, source=np.asarray(f(x)), D_xx_coefficients=np.ones(x.shape[:2]),
                             D_yy_coefficients=np.ones(x.shape[:2]))

        def run():
            hps.build_solver(pde)
            return [hps.solve(pde, dom.get_adaptive_boundary_data_lst(lambda b: b[:, 0].copy()))]

        return run
    dom = hps.Domain(p=12, q=10, root=hps.DiscretizationNode2D(-1.0, 1.0, -1.0, 1.0), L=3)
    x = dom.interior_points
    iti = "iti" in kind
    kw = dict(D_xx_coefficients=np.ones(x.shape[:2]), D_yy_coefficients=np.ones(x.shape[:2]),
              I_coefficients=(20.0 if iti else 1.0) * np.ones(x.shape[:2]))
    if iti:
        kw.update(use_ItI=True, eta=4.0)
    f = np.sin(x[..., 0]) + x[..., 1]
    g = rng.standard_normal(dom.boundary_points.shape[0]) * (1 + (1j if iti else 0))
    nosource = "nosource" in kind
    pde = hps.PDEProblem(dom, source=None if nosource else f, **kw)

    def run():
        top = hps.build_solver(pde, return_top_T=True)
        return [top, hps.solve(pde, g, source=f if nosource else None)]

    return run


@pytest.mark.parametrize("kind", ["dtn", "iti", "nosource dtn", "nosource iti", "adaptive"])
@pytest.mark.parametrize("which", [0, -1, 1])
def test_every_stage_goes_back_to_the_level(cuda, monkeypatch, kind, which):
    """One refined merge call (the first, the last, the second) marked as not refined,
    with NaN for its outputs: the results are the unmarked ones, to the 1e-11 between
    a refined and an eliminated inverse."""
    run = _stage(kind)
    calls, real = _record(monkeypatch)
    ref = run()
    n = len(calls)
    monkeypatch.undo()
    count = [0]
    refined_calls = []

    def level(T, h, maps, **kw):
        lst = kw.get("refined")
        before = 0 if lst is None else len(lst)
        out = real(T, h, maps, **kw)
        if lst is not None and len(lst) > before:       # large enough to be refined
            refined_calls.append(count[0])
            if target is not None and count[0] == target:
                lst[-1].fill_(nat.INFO_NOT_REFINED)
                for t in out:
                    if t is not None:
                        t.fill_(float("nan"))
        count[0] += 1
        return out

    target = None
    monkeypatch.setattr(st, "merge_level_dtn", level)
    run()
    assert len(refined_calls) >= 2 and count[0] == n
    target = refined_calls[which]
    count[0] = 0
    got = run()
    assert count[0] > n
    for a, b in zip(got, ref):
        a, b = torch.as_tensor(a), torch.as_tensor(b)
        assert float((a - b).abs().max()) <= 1e-11 * float(b.abs().max())
