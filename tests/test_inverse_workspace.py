"""Workspace of the batched inverses: what is asked for is what the kernels use."""

import numpy as np
import pytest
import torch

from jaxhps_gb300 import _build
from jaxhps_gb300 import _native as nat

F64, F32, C128, C64 = 0, 1, 2, 3
TYPES = {F64: torch.float64, F32: torch.float32, C128: torch.complex128, C64: torch.complex64}


@pytest.mark.parametrize("dtype,size,panels", [(F64, 8, 4), (F32, 4, 3), (C128, 16, 4), (C64, 8, 3)])
@pytest.mark.parametrize("n", [300, 777])
def test_panels_that_are_formed(dtype, size, panels, n):
    """The tableau, the panel, U and G, and H for the FP64 types only (32 columns or rows
    each); the rest is E, pivots, flags and the panels' proposal slots."""
    _build.build()
    lib = nat.load_library()
    one = lib.hps_inverse_workspace_size(dtype, n, 101) - lib.hps_inverse_workspace_size(dtype, n, 100)
    least = size * n * n + panels * 32 * n * size
    rest = 1024 * size + 16 * n + 2 * max(n // 16, 16) * (12 + 32 * size) + 4096
    assert least <= one <= least + rest


@pytest.mark.gpu
@pytest.mark.parametrize("entry", ["hps_inverse_batched", "hps_inverse_interface"])
@pytest.mark.parametrize("dtype", list(TYPES))
@pytest.mark.parametrize("n,batch", [(140, 5), (256, 3), (300, 160), (700, 1)])
def test_nothing_is_written_behind_it(cuda, entry, dtype, n, batch):
    lib, dt = nat.lib(), TYPES[dtype]
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((batch, n, n), dtype=dt, device="cuda", generator=g) + 3 * n ** 0.5 * torch.eye(n, dtype=dt, device="cuda")
    X = torch.empty_like(A)
    info = torch.full((batch,), 7, dtype=torch.int32, device="cuda")
    size = lib.hps_inverse_workspace_size(dtype, n, batch)
    ws = torch.full((size + 4096,), 0x5a, dtype=torch.uint8, device="cuda")
    assert getattr(lib, entry)(dtype, n, A.data_ptr(), n, n * n, X.data_ptr(), n, n * n, batch, info.data_ptr(),
                               ws.data_ptr(), size, nat.stream_ptr()) == 0
    assert not info.any() and bool((ws[size:] == 0x5a).all())
    eps = 2.0 ** -53 if dtype in (F64, C128) else 2.0 ** -24
    cond = float(torch.linalg.cond(A[0], np.inf))
    err = (X @ A - torch.eye(n, dtype=dt, device="cuda")).abs().max()
    assert float(err) <= 4 * n * cond * eps
