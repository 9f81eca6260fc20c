"""The FP64 leaf stages and the impedance merges issue device work only, so that
they can be captured in a CUDA graph (their inverses are then eliminated: the
refinement's status words cannot be read while capturing)."""

import pytest
import torch

import jaxhps_gb300 as hps
from jaxhps_gb300 import _iti
from jaxhps_gb300 import _stages as st

pytestmark = pytest.mark.gpu


def _pde(iti):
    dom = hps.Domain(p=11, q=9, root=hps.DiscretizationNode2D(-1.0, 1.0, -1.0, 1.0), L=2)
    x = torch.as_tensor(dom.interior_points, device="cuda")
    one = torch.ones(x.shape[:2], dtype=torch.float64, device="cuda")
    kw = dict(D_xx_coefficients=one, D_yy_coefficients=one.clone(), I_coefficients=4.0 * one)
    if iti:
        kw.update(use_ItI=True, eta=4.0)
    return hps.PDEProblem(dom, source=torch.sin(3 * x[..., 0]) + x[..., 1], **kw)


@pytest.mark.parametrize("stage", ["dtn leaf", "iti leaf", "iti merge"])
def test_stages_in_a_graph(cuda, stage):
    """n = 81 and 121 (leaves), 18 to 72 (two-colour merges).  Eliminated or refined, both
    are FP64 inverses and agree to 1e-11 of the largest entry."""
    pde = _pde(stage.startswith("iti"))
    leaf = st.local_solve_stage_uniform_2D_ItI if pde.use_ItI else st.local_solve_stage_uniform_2D_DtN
    Y, T, v, h = leaf(pde)

    def run():
        if stage.endswith("leaf"):
            return list(leaf(pde))
        S, g = _iti.merge_stage_uniform_2D_ItI(T, h, l=2)
        return [*S, *g]

    ref = run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    for t in out:
        t.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(out, ref):
        assert float((a - b).abs().max()) <= 1e-11 * float(b.abs().max())
