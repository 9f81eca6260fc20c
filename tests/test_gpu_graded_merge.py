"""FP64 merges whose interface rows have several scales (csrc/hps_kernels.cu,
balance_rows), as the children's DtN rows have where their panels differ in size."""

import numpy as np
import pytest
import torch

from jaxhps_gb300 import _native as nat
from jaxhps_gb300 import _stages as st
from jaxhps_gb300._index_maps import oct_merge_maps_dtn, quad_merge_maps_dtn

pytestmark = pytest.mark.gpu


def _merge(T, h, maps):
    """Every output, by refined inverses and again by elimination where one was not."""
    for refined in ([], None):
        out = st.merge_level_dtn(T, h, maps, keep_D_inv=True, keep_BD_inv=True, refined=refined)
        if not st.unrefined(refined):
            return [x.cpu().numpy() for x in out]


@pytest.mark.parametrize("rects", [True, False])
@pytest.mark.parametrize("kind,q,nm,ns", [("quad", 9, 5, 1), ("quad", 28, 3, 12), ("oct", 5, 2, 3)])
@pytest.mark.parametrize("k", [-40, 3, 12, 20, 40])
def test_interface_rows_of_several_scales(cuda, monkeypatch, kind, q, nm, ns, k, rects):
    """The rows of both children at one interface point in 16 times 2^k: S, g~, T and h
    are those without it, D^-1's and B D^-1's columns 2^-k times.  n_int = 36, 112 and
    300: below and above what is refined.  Both sides carry n cond(D) 2^-53 of the
    largest entry, cond(D) <= 4: children of 4 I + random with row sums below 1."""
    monkeypatch.setattr(st, "_RECTS", rects)
    maps = {"quad": quad_merge_maps_dtn, "oct": lambda n: oct_merge_maps_dtn(n * n)}[kind](q)
    rng = np.random.default_rng(q)
    T = rng.standard_normal((nm, maps.nch, maps.nb, maps.nb)) / (4 * maps.nb) + 4 * np.eye(maps.nb)
    h = rng.standard_normal((nm, maps.nch, maps.nb, ns))
    r = np.where(np.arange(maps.n_int) % 16 == 5, 2.0 ** k, 1.0)
    Ts, hs = T.copy(), h.copy()
    for i in range(maps.n_int):
        for c, l in zip(maps.int_c[i], maps.int_l[i]):
            Ts[:, c, l] *= r[i]
            hs[:, c, l] *= r[i]
    dev = lambda a: torch.as_tensor(a.reshape(nm * maps.nch, *a.shape[2:]), device="cuda")  # noqa: E731
    ref = _merge(dev(T), dev(h), maps)
    got = _merge(dev(Ts), dev(hs), maps)
    got[4], got[5] = got[4] * r, got[5] * r
    tol = 2 * maps.n_int * 4 * 2.0 ** -53
    for name, a, b in zip(("S", "g", "T", "h", "D_inv", "BD_inv"), got, ref):
        assert np.abs(a - b).max() <= tol * np.abs(b).max(), (name, float(np.abs(a - b).max() / np.abs(b).max()), tol)


def test_rows_of_zeros_and_infinities_stay_in_their_merge(cuda):
    maps = quad_merge_maps_dtn(20)
    rng = np.random.default_rng(0)
    T = rng.standard_normal((4, maps.nch, maps.nb, maps.nb)) / (4 * maps.nb) + 4 * np.eye(maps.nb)
    bad = T.copy()
    for c, l in zip(maps.int_c[0], maps.int_l[0]):
        bad[0, c, l] = 0.0                    # the first row, which the others are compared with
    for c, l in zip(maps.int_c[33], maps.int_l[33]):
        bad[2, c, l, 3] = np.inf
    run = lambda t: st.merge_level_dtn(torch.as_tensor(t.reshape(-1, *t.shape[2:]), device="cuda"), None, maps)[0]  # noqa: E731
    a, b = run(bad), run(T)
    assert torch.equal(a[1], b[1]) and torch.equal(a[3], b[3])
    assert nat.load_library().hps_gemm_tc_status() == 0
