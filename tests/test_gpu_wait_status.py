"""Every public call that runs products on the tensor-core kernels reads their
timeout flag before it returns: a set flag raises there, and not in a later
call.  The flag's reading is replaced on the host (no wait runs out here)."""

import numpy as np
import pytest

import jaxhps_gb300 as hps
from jaxhps_gb300 import _native as nat

pytestmark = pytest.mark.gpu


class _TimedOut:
    """The library with its flag set once."""

    def __init__(self, lib):
        self._lib, self.flag = lib, 1

    def __getattr__(self, name):
        return getattr(self._lib, name)

    def hps_gemm_tc_status_reset(self):
        flag, self.flag = self.flag, 0
        return flag


def _pde(iti=False):
    dom = hps.Domain(p=8, q=6, root=hps.DiscretizationNode2D(-1.0, 1.0, -1.0, 1.0), L=2)
    x = dom.interior_points
    ones = np.ones(x.shape[:2])
    kw = dict(D_xx_coefficients=ones, D_yy_coefficients=ones, I_coefficients=9.0 * ones)
    if iti:
        kw.update(use_ItI=True, eta=3.0)
    return hps.PDEProblem(dom, source=np.sin(x[..., 0]), **kw), dom.boundary_points[:, 0] + (0j if iti else 0.0)


def _calls():
    dom2 = hps.Domain(p=8, q=6, root=hps.DiscretizationNode2D(-1.0, 1.0, -1.0, 1.0), L=1)
    dom3 = hps.Domain(p=6, q=4, root=hps.DiscretizationNode3D(-1.0, 1.0, -1.0, 1.0, -1.0, 1.0), L=1)
    s = np.linspace(-1.0, 1.0, 7)

    def down(iti):
        pde, g = _pde(iti)
        hps.upward_pass_subtree(pde)
        return lambda: hps.downward_pass_subtree(pde, g)

    def solve():
        pde, g = _pde()
        hps.build_solver(pde)
        return lambda: hps.solve(pde, g)

    return {
        "build_solver": lambda: lambda: hps.build_solver(_pde()[0]),
        "solve": solve,
        "solve_subtree": lambda: lambda: hps.solve_subtree(*_pde()),
        "solve_subtree iti": lambda: lambda: hps.solve_subtree(*_pde(True)),
        "upward_pass_subtree": lambda: lambda: hps.upward_pass_subtree(_pde()[0]),
        "downward_pass_subtree": lambda: down(False),
        "downward_pass_subtree iti": lambda: down(True),
        "interp 2D": lambda: lambda: dom2.interp_to_interior_points(np.ones((7, 7)), s, s),
        "interp 3D": lambda: lambda: dom3.interp_to_interior_points(np.ones((7, 7, 7)), s, s, s),
    }


@pytest.mark.parametrize("name", ["build_solver", "solve", "solve_subtree", "solve_subtree iti", "upward_pass_subtree",
                                  "downward_pass_subtree", "downward_pass_subtree iti", "interp 2D", "interp 3D"])
def test_a_set_flag_raises_in_the_call(cuda, monkeypatch, name):
    call = _calls()[name]()
    real = nat.lib()
    fake = _TimedOut(real)
    monkeypatch.setattr(nat, "lib", lambda: fake)
    with pytest.raises(nat.DeviceWaitTimeout):
        call()
    call()                      # the flag was cleared: the next call is sound
    monkeypatch.undo()
    assert real.hps_gemm_tc_status() == 0


@pytest.mark.parametrize("call", [lambda pde, g: hps.solve_subtree(pde, g), lambda pde, g: hps.upward_pass_subtree(pde)])
def test_a_singular_leaf_raises_in_the_subtree_calls(cuda, call):
    pde, g = _pde()
    x = pde.domain.interior_points
    zero = np.ones(x.shape[:2])
    zero[5] = 0.0
    pde = hps.PDEProblem(pde.domain, source=np.ones(x.shape[:2]), D_xx_coefficients=zero, D_yy_coefficients=zero,
                         I_coefficients=zero)
    with pytest.raises(nat.SingularPivotError):
        call(pde, g)
