"""FP64 and complex128 products from 8-bit digits on the tensor cores
(csrc/gemm_f64_tc.cu) at the edges of its 128 x 64 / 128 x 16 tiles, its
stages of 16 and chunks of 128 steps, with odd leading dimensions, broadcast
operands, scaled and special values.

Reference: the product in numpy's long double.  Tolerance per entry: one
rounding of the result and one of the addition of C (2^-52 |r|), and the
truncation: operands cut below 2^-61 of their row's or column's largest entry
and digit products below the eighth weight, together at most 2^-56 per step
of the product of the two largest entries (complex: four real products)."""

import numpy as np
import pytest
import torch

from jaxhps_gb300 import _native as nat

pytestmark = pytest.mark.gpu

NONE, RULE, ALL = 0, 1, 2


@pytest.fixture
def policy(cuda):
    lib = nat.load_library()
    yield lib.hps_gemm_policy
    lib.hps_gemm_policy(RULE)


def _draw(rng, shape, cplx, spread):
    x = rng.standard_normal(shape) * 10.0 ** (spread * rng.uniform(-0.5, 0.5, shape))
    return x + 1j * rng.standard_normal(shape) if cplx else x


def _exact(A, B):
    wide = np.clongdouble if np.iscomplexobj(A) else np.longdouble
    return np.matmul(A.astype(wide), B.astype(wide))


def _check(got, A, B, alpha, C):
    if got.shape[0] > 3:   # the first and the last matrices of a large batch: long double is slow
        pick = [0, got.shape[0] - 1]
        got, B, C = got[pick], B[pick], None if C is None else C[pick]
        A = A if A.shape[0] == 1 else A[pick]
    ref = alpha * _exact(A, B) + (0 if C is None else C)
    am = np.maximum(np.abs(A.real), np.abs(A.imag)).max(-1)[..., :, None]
    bm = np.maximum(np.abs(B.real), np.abs(B.imag)).max(-2)[..., None, :]
    k = A.shape[-1] * (4 if np.iscomplexobj(A) else 1)
    tol = 2.0 ** -52 * np.abs(ref) + abs(alpha) * k * 2.0 ** -56 * am * bm
    assert (np.abs(got - ref) <= tol).all(), float((np.abs(got - ref) / tol).max())


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("M,N,K,batch,pad,spread", [
    (1, 1, 1, 1, 0, 0), (1, 9, 16, 3, 1, 0), (127, 16, 17, 2, 0, 4), (128, 17, 31, 1, 1, 0), (129, 63, 127, 2, 0, 2),
    (128, 64, 128, 2, 0, 0), (130, 65, 129, 1, 3, 6), (257, 33, 300, 2, 1, 0), (56, 8, 256, 40, 0, 2),
    (196, 56, 196, 160, 0, 0), (300, 130, 260, 1, 2, 8)])
def test_products_at_tile_edges(policy, M, N, K, batch, pad, spread, cplx):
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    dt = torch.complex128 if cplx else torch.float64
    A, B = _draw(rng, (batch, M, K + pad), cplx, spread), _draw(rng, (batch, K, N + pad), cplx, spread)
    C = _draw(rng, (batch, M, N), cplx, spread)
    At, Bt, Ct = (torch.as_tensor(t, dtype=dt, device="cuda") for t in (A, B, C))
    a, b = At[..., :K], Bt[..., :N]
    policy(ALL)
    for alpha, c, left in ((1.0, None, a), (-1.0, Ct, a), (0.375, Ct, a[0])):
        D = torch.full((batch, M, N + pad), float("nan"), dtype=dt, device="cuda")[..., :N]
        if c is None:
            nat.gemm(left, b, D, alpha)
        else:
            nat.gemm(left, b, D, alpha, 1.0, Cmat=c)
        ah = A[..., :K] if left is a else A[:1, :, :K]
        _check(D.cpu().numpy(), ah, B[..., :N], alpha, None if c is None else C)
    assert nat.load_library().hps_gemm_tc_status() == 0


@pytest.mark.parametrize("cplx", [False, True])
def test_infinities_nan_zero_and_tiny_rows(policy, cplx):
    """Rows and columns that cannot be scaled to integers give what the
    multiply-add chain gives; rows of zeros give exact zeros."""
    rng = np.random.default_rng(5)
    dt = torch.complex128 if cplx else torch.float64
    A, B = _draw(rng, (150, 90), cplx, 0), _draw(rng, (90, 70), cplx, 0)
    A[3, 5], A[7, 8], A[20], A[21], A[30] = np.inf, np.nan, A[20] * 1e-300, A[21] * 1e-318, A[30] * 1e150
    A[10], A[11] = 0.0, -0.0
    B[4, 6], B[:, 9], B[:, 11] = -np.inf, 0.0, B[:, 11] * 1e200
    At, Bt = torch.as_tensor(A, dtype=dt, device="cuda"), torch.as_tensor(B, dtype=dt, device="cuda")
    out = []
    for pol in (NONE, ALL):
        policy(pol)
        D = torch.empty((150, 70), dtype=dt, device="cuda")
        nat.gemm(At, Bt, D)
        out.append(torch.view_as_real(D).cpu().numpy() if cplx else D.cpu().numpy())
    chain, digits = out
    assert np.array_equal(np.isnan(chain), np.isnan(digits)) and np.array_equal(np.isinf(chain), np.isinf(digits))
    fin = np.isfinite(chain)
    keep = [c for c in range(70) if c != 6]
    assert (digits[10:12][:, keep] == 0).all()
    row = np.abs(np.where(fin, chain, 0)).max(1, keepdims=True) if not cplx else \
        np.abs(np.where(fin, chain, 0)).max((1, 2), keepdims=True)
    # the chain's own rounding: 90 steps (180 real ones) of 2^-53 of the partial sums
    assert (np.abs(np.where(fin, chain - digits, 0)) <= 400 * 2.0 ** -53 * 4 * row).all()


@pytest.mark.parametrize("rows", [0, 8])
@pytest.mark.parametrize("K", [49, 196, 700])
def test_no_less_exact_than_the_chain(policy, K, rows):
    """Normal entries, rows of A and columns of B scaled over 0 or 8 decades
    (not the single entries: a product whose large entries meet small ones
    only is held to the bound at the top of this file, not to the chain's)."""
    rng = np.random.default_rng(K + rows)
    A, B = _draw(rng, (190, K), False, 0), _draw(rng, (K, 70), False, 0)
    A *= 10.0 ** (rows * rng.uniform(-0.5, 0.5, (190, 1)))
    B *= 10.0 ** (rows * rng.uniform(-0.5, 0.5, (1, 70)))
    ref, scale = _exact(A, B), np.abs(A) @ np.abs(B)
    At, Bt = torch.as_tensor(A, device="cuda"), torch.as_tensor(B, device="cuda")
    err = []
    for pol in (NONE, ALL):
        policy(pol)
        D = torch.empty((190, 70), dtype=torch.float64, device="cuda")
        nat.gemm(At, Bt, D)
        err.append((np.abs(D.cpu().numpy() - ref) / scale).astype(np.float64))
    assert np.sqrt((err[1] ** 2).mean()) <= np.sqrt((err[0] ** 2).mean())
    assert err[1].max() <= err[0].max()


@pytest.mark.parametrize("p,q", [(13, 11), (16, 14)])
def test_leaf_operators_no_less_exact_than_the_chain(policy, p, q):
    """Y and T of variable-coefficient leaves against long double."""
    import jaxhps_gb300 as hps
    from jaxhps_gb300 import _stages as st

    dom = hps.Domain(p=p, q=q, root=hps.DiscretizationNode2D(-1.0, 0.0, -1.0, 0.0), L=2)
    x = dom.interior_points
    kw = dict(D_xx_coefficients=1 + 0.3 * np.cos(x[..., 0]) ** 2, D_yy_coefficients=np.ones(x.shape[:2]),
              D_xy_coefficients=0.2 * np.sin(x[..., 0]), I_coefficients=1 + 0.5 * np.exp(-((x + 0.5) ** 2).sum(-1) / 0.04))
    pde = hps.PDEProblem(dom, source=np.ones(x.shape[:2]), **kw)
    n_cb = pde.P.shape[0]
    cs, ops = pde.active_coefficients()
    leaves = (0, 7, 15)
    wide = np.longdouble
    ref = []
    for l in leaves:
        A = sum(c[l][:, None].astype(wide) * o.astype(wide) for c, o in zip(cs, ops))[n_cb:]
        M = np.concatenate([A[:, n_cb:], -A[:, :n_cb] @ pde.P.astype(wide)], 1)
        n = M.shape[0]
        for k in range(n):   # Gauss-Jordan with row exchanges
            r = k + int(np.argmax(np.abs(M[k:, k])))
            M[[k, r]] = M[[r, k]]
            M[k] /= M[k, k]
            f = M[:, k].copy()
            f[k] = 0
            M[:, k:] -= f[:, None] * M[k, k:]
        Y = np.concatenate([pde.P.astype(wide), M[:, n:]])
        ref.append((Y, pde.Q.astype(wide) @ Y))
    err = []
    for pol in (NONE, RULE):
        policy(pol)
        Y, T, _, _ = st.local_solve_stage_uniform_2D_DtN(pde)
        rel = [[np.linalg.norm((g[l].cpu().numpy() - r).astype(float)) / np.linalg.norm(r.astype(float))
                for g, r in zip((Y, T), rr)] for l, rr in zip(leaves, ref)]
        err.append(np.sqrt((np.array(rel) ** 2).mean(0)))
    assert (err[1] <= err[0]).all(), err


@pytest.mark.parametrize("N", [1, 2, 8])
def test_few_columns_either_way(policy, N):
    """The dispatch rule's two sides for N <= 8 agree to rounding."""
    rng = np.random.default_rng(N)
    A, B = _draw(rng, (700, 196, 196), False, 0), _draw(rng, (700, 196, N), False, 0)
    At, Bt = torch.as_tensor(A, device="cuda"), torch.as_tensor(B, device="cuda")
    out = []
    for pol in (NONE, RULE):
        policy(pol)
        D = torch.empty((700, 196, N), dtype=torch.float64, device="cuda")
        nat.gemm(At, Bt, D)
        out.append(D)
    scale = At.abs() @ Bt.abs()
    assert float(((out[0] - out[1]).abs() / scale).max()) <= 196 * 2.0 ** -53


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("M,N,K,batch,pad", [(196, 196, 4, 256, 0), (196, 196, 16, 256, 0), (196, 196, 32, 256, 0),
                                             (130, 10, 20, 400, 0), (196, 196, 16, 256, 1), (128, 64, 17, 400, 3)])
def test_many_short_tiles_with_a_c(policy, M, N, K, batch, pad, cplx):
    """Several tiles a CTA whose operands wait in the ring while sums are rounded
    and C is read, every matrix of the batch and several runs: even and odd rows
    (tensor-map boxes and single copies).  Against torch's FP64 product: K + 2
    roundings of the sum of the magnitudes on its side, 2^-56 of the row's and
    column's largest per step here, both below 2 (K + 2) 2^-53 of the bound."""
    g = torch.Generator(device="cuda").manual_seed(K)
    dt = torch.complex128 if cplx else torch.float64
    A, B, C = (torch.randn((batch, m, n + pad), dtype=dt, device="cuda", generator=g)[..., :n]
               for m, n in ((M, K), (K, N), (M, N)))
    ref = A @ B + C
    am = A.abs().amax(-1, keepdim=True)
    bm = B.abs().amax(-2, keepdim=True)
    tol = 2 * (K + 2) * 2.0 ** -53 * (4 if cplx else 1) * (K * am * bm + C.abs())
    policy(ALL)
    for _ in range(3):
        D = C.clone()
        nat.gemm(A, B, D, 1.0, 1.0, Cmat=D)
        assert bool(((D - ref).abs() <= tol).all())
