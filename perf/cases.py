"""The work that a user of this package has it do, as cases to time.

A case is one call chain through the public entry points: ``build_solver`` +
``solve`` on a uniform quadtree (DtN or impedance maps), on a uniform octree
or on an adaptive octree that is meshed first; ``solve`` of new sources with
the operators of an earlier build; and the interpolation of a solution to a
rectangular grid.  ``exact`` solves the same discrete problems by pairwise
merges with ``torch.linalg`` in 64 bits.
"""

import math

import numpy as np
import torch

import jaxhps_gb300 as hps

DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def _case(name, kind, L, p, precision, nsrc=1, q=None, terms="helm", top=False, host=True, **more):
    c = dict(name=name, kind=kind, L=L, p=p, q=p - 2 if q is None else q, precision=precision, nsrc=nsrc,
             terms=terms, top=top, host=host)
    c.update(more)
    return c


def listed():
    return [
        # the first example of a new user, and the unit of a parameter study on a small problem: latency
        _case("dtn2d_f64_L3_p8", "dtn2d", 3, 8, "float64"),
        # variable coefficients in every term, odd sizes, several sources, default precision
        _case("dtn2d_f64_L4_p13_full", "dtn2d", 4, 13, "float64", nsrc=3, terms="full", top=True),
        # the usual 2D problem at the default precision
        _case("dtn2d_f64_L6_p16", "dtn2d", 6, 16, "float64"),
        # one source, mixed precision: an ordinary 2D problem
        _case("dtn2d_mixed_L5_p16", "dtn2d", 5, 16, "mixed"),
        # the benchmark's configuration: 16,384 leaves, 64 sources, the result kept on the device
        _case("dtn2d_mixed_L7_p16_64", "dtn2d", 7, 16, "mixed", nsrc=64, host=False),
        # scattering: the interior impedance problem whose top map is coupled to an exterior one
        _case("iti2d_f64_L5_p16_top", "iti2d", 5, 16, "float64", top=True, wave=20.0),
        # the same at the size where mixed precision is used
        _case("iti2d_mixed_L6_p16", "iti2d", 6, 16, "mixed", wave=40.0),
        # 3D at the default precision: 64 leaves of 1,000 points
        _case("dtn3d_f64_L2_p10", "dtn3d", 2, 10, "float64"),
        # the largest 3D configuration: 512 leaves
        _case("dtn3d_mixed_L3_p10", "dtn3d", 3, 10, "mixed"),
        # a wavefront: adaptive meshing, then build and solve on the uneven tree
        _case("adaptive3d_f64_p8", "adaptive3d", 0, 8, "float64", tol=1e-3, sharp=10.0, centre=-0.05),
        # many solves with one build: new sources and boundary data, as in time stepping or an inverse problem
        _case("resolve2d_f64_L6_p16_8", "resolve2d", 6, 16, "float64", nsrc=8),
        # the solution on a rectangular grid, for plots and for coupling to other codes
        _case("interp2d_L6_p16", "interp2d", 6, 16, "float64", nx=512, ny=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges (orders, depths, sources, terms, precisions)."""
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["dtn2d", "dtn2d", "dtn2d", "iti2d", "dtn3d", "adaptive3d", "resolve2d", "interp2d"])
        precision = rng.choice(["float64", "mixed"])
        p = rng.randint(7, 16)
        q = p - 3 if precision == "float64" and rng.random() < 0.4 else p - 2
        nsrc = _log_int(rng, 1, 64)
        if kind == "dtn2d":
            c = _case("", kind, rng.randint(1, 6), p, precision, nsrc=nsrc, q=q, terms=rng.choice(["helm", "full"]),
                      top=precision == "float64" and rng.random() < 0.3)
        elif kind == "iti2d":
            c = _case("", kind, rng.randint(2, 6), max(p, 10), precision, nsrc=_log_int(rng, 1, 4),
                      top=rng.random() < 0.5)
            c["wave"] = float(rng.randint(4, 6)) * 2.0 ** (c["L"] - 2)
        elif kind == "dtn3d":
            p = rng.randint(6, 10)
            c = _case("", kind, rng.randint(1, 3), p, precision, nsrc=_log_int(rng, 1, 4))
        elif kind == "adaptive3d":
            p = rng.choice([6, 8, 10])
            c = _case("", kind, 0, p, "float64", tol=10.0 ** rng.uniform(-3.0, -2.0), sharp=rng.uniform(5.0, 10.0),
                      centre=rng.uniform(-0.07, -0.03))
        elif kind == "resolve2d":
            c = _case("", kind, rng.randint(2, 6), p, "float64", nsrc=nsrc, q=q)
        else:
            c = _case("", kind, rng.randint(2, 6), p, "float64", nx=_log_int(rng, 33, 700), ny=_log_int(rng, 33, 700))
        if _cost(c) <= most:
            del c["name"]
            return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _bumps(x, gen, n, width, dtype=torch.float64):
    """Sum of n Gaussians with seeded centres and amplitudes at the points x (..., d)."""
    d = x.shape[-1]
    z = torch.as_tensor(gen.uniform(-0.8, 0.8, (n, d)), device=x.device)
    a = gen.uniform(0.3, 1.0, n)
    out = torch.zeros(x.shape[:-1], dtype=dtype, device=x.device)
    for k in range(n):
        out += float(a[k]) * torch.exp(-((x - z[k]) ** 2).sum(-1) / width ** 2)
    return out


def _coefficients(case, x, gen):
    """{term: values at the leaf points}."""
    ones = torch.ones(x.shape[:2], dtype=torch.float64, device=x.device)
    if case["kind"] == "iti2d":
        k = case["wave"]
        return {"D_xx": ones, "D_yy": ones.clone(), "I": k * k * (1.0 + 0.25 * _bumps(x, gen, 6, 0.15))}
    out = {"D_xx": ones, "D_yy": ones.clone()}
    if x.shape[-1] == 3:
        out["D_zz"] = ones.clone()
    out["I"] = 1.0 + 0.25 * _bumps(x, gen, 4, 0.2)
    if case["terms"] == "full":
        out["D_xx"] = 1.0 + 0.3 * torch.cos(x[..., 0] + gen.uniform(-1, 1)) ** 2
        out["D_yy"] = 1.0 + 0.3 * torch.sin(x[..., 1] + gen.uniform(-1, 1)) ** 2
        out["D_xy"] = 0.2 * torch.sin(x[..., 0]) * torch.cos(x[..., 1])
        out["D_x"] = 0.3 * torch.cos(2 * x[..., 1])
        out["D_y"] = 0.2 * x[..., 0] * x[..., 1]
    return out


def _fields(case, x, b, gen):
    """(coefficients, source, boundary data) on the leaf points x and the boundary points b."""
    coeffs = _coefficients(case, x, gen)
    ns = case["nsrc"]
    if case["kind"] == "iti2d":
        th = gen.uniform(0, 2 * np.pi, ns)
        k = case["wave"]
        contrast = coeffs["I"] - k * k
        f = torch.stack([-contrast * torch.exp(1j * k * (math.cos(t) * x[..., 0] + math.sin(t) * x[..., 1]))
                         for t in th], -1)
        g = torch.stack([torch.exp(1j * (math.cos(t) * b[:, 0] + math.sin(t) * b[:, 1])) for t in th], -1)
    else:
        amp = gen.uniform(-1, 1, ns)
        f = torch.empty(x.shape[:2] + (ns,), dtype=torch.float64, device=x.device)
        for j in range(ns):
            f[..., j] = _bumps(x, gen, 3, 0.15) + float(amp[j])
        lin = gen.uniform(-1, 1, (2, ns))
        g = torch.stack([float(lin[0, j]) * (b[:, 0] ** 2 - b[:, 1] ** 2) + float(lin[1, j]) * torch.sin(b[:, 0] + b[:, 1])
                         for j in range(ns)], -1)
    if ns == 1:
        f, g = f[..., 0].contiguous(), g[..., 0].contiguous()
    return coeffs, f, g


def _domain(case):
    L, p, q = case["L"], case["p"], case["q"]
    if case["kind"] == "dtn3d":
        return hps.Domain(p=p, q=q, root=hps.DiscretizationNode3D(-1.0, 1.0, -1.0, 1.0, -1.0, 1.0), L=L)
    return hps.Domain(p=p, q=q, root=hps.DiscretizationNode2D(-1.0, 1.0, -1.0, 1.0), L=L)


def _inputs(case, seed, x, b):
    return _fields(case, x, b, np.random.default_rng(int(seed)))


class _Front:
    """u = arctan(k (|x - c| - R)) and its Laplacian, on arrays or tensors."""

    def __init__(self, k, c, R):
        self.k, self.c, self.R = k, c, R

    def _r(self, x):
        xp = torch if isinstance(x, torch.Tensor) else np
        return xp, xp.sqrt((x[..., 0] - self.c[0]) ** 2 + (x[..., 1] - self.c[1]) ** 2 + (x[..., 2] - self.c[2]) ** 2)

    def u(self, x):
        xp, r = self._r(x)
        return xp.arctan(self.k * (r - self.R))

    def f(self, x):
        _, r = self._r(x)
        s = self.k * (r - self.R)
        return -2 * self.k * self.k * s / (1 + s * s) ** 2 + 2 * self.k / ((1 + s * s) * r)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "adaptive3d":
        gen = np.random.default_rng(int(seed))
        return dict(case=case, front=_Front(case["sharp"], (case["centre"],) * 3, 0.6), amp=gen.uniform(0.2, 1.0, 2))
    dom = _domain(case)
    x = torch.as_tensor(dom.interior_points, device=DEV)
    b = torch.as_tensor(dom.boundary_points, device=DEV)
    if kind == "interp2d":
        gen = np.random.default_rng(int(seed))
        s = _bumps(x, gen, 8, 0.3)
        ex, ey = _eval_points(case)
        return dict(case=case, dom=dom, samples=s, ex=ex, ey=ey)
    coeffs, f, g = _inputs(case, seed, x, b)
    kw = {k + "_coefficients": v for k, v in coeffs.items()}
    if kind == "iti2d":
        kw.update(use_ItI=True, eta=float(case["wave"]))
    pde = hps.PDEProblem(dom, source=None if kind == "resolve2d" else f, **kw)
    if kind == "resolve2d":
        hps.build_solver(pde)
    return dict(case=case, pde=pde, f=f, g=g)


def _eval_points(case):
    # inside the domain, off the leaf interfaces
    nx, ny = case["nx"], case["ny"]
    return (np.linspace(-1, 1, nx + 2)[1:-1] * 0.99 + 0.00123, np.linspace(-1, 1, ny + 2)[1:-1] * 0.99 - 0.00217)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "adaptive3d":
        return _run_adaptive(case, state["front"], state["amp"])
    if kind == "interp2d":
        vals, target = state["dom"].interp_from_interior_points(state["samples"], state["ex"], state["ey"])
        return {"values": vals, "points": target}
    host = "cpu" if case["host"] else None
    if kind == "resolve2d":
        return {"u": hps.solve(state["pde"], state["g"], source=state["f"], host_device=host)}
    pde = state["pde"]
    top = hps.build_solver(pde, return_top_T=case["top"], precision=case["precision"])
    out = {"u": hps.solve(pde, state["g"], host_device=host)}
    if case["top"]:
        out["top"] = top
    return out


def _run_adaptive(case, front, amp):
    """Meshes the front, then solves for it in a medium and with boundary data that come with the inputs."""
    root = hps.DiscretizationNode3D(0.0, 1.0, 0.0, 1.0, 0.0, 1.0)
    dom = hps.Domain.from_adaptive_discretization(p=case["p"], q=case["q"], root=root, f=front.f, tol=case["tol"])
    x = dom.interior_points
    ones = np.ones(x.shape[:2])
    medium = amp[0] * np.exp(-((x - 0.4) ** 2).sum(-1) / 0.1)
    pde = hps.PDEProblem(dom, source=front.f(x), D_xx_coefficients=ones, D_yy_coefficients=ones,
                         D_zz_coefficients=ones, I_coefficients=medium)
    hps.build_solver(pde)
    return {"u": hps.solve(pde, dom.get_adaptive_boundary_data_lst(lambda b: amp[1] * front.u(b))), "points": x}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------


def _tree_flops(d, L, ni, npts, nb_leaf, nsrc):
    """Leaf solves, quad / oct Schur complements by two-way merges, down pass: real multiply-adds x 2."""
    leaves = (2 ** d) ** L
    fl = leaves * (2.0 / 3.0 * ni ** 3 + 2.0 * ni * ni * (nb_leaf + nsrc) + 2.0 * nb_leaf * npts * (nb_leaf + 2 * nsrc))
    face = nb_leaf / (2.0 * d)
    dims = [1] * d
    count = leaves
    for _ in range(L):
        for a in range(d):
            count //= 2
            m = face * np.prod([dims[k] for k in range(d) if k != a])
            dims[a] *= 2
            area = face * 2 * sum(np.prod([dims[k] for k in range(d) if k != j]) for j in range(d))
            fl += count * (2.0 / 3.0 * m ** 3 + 2.0 * m * m * (area + nsrc) + 2.0 * m * area * area / 2 + 4.0 * m * area * nsrc)
    return fl


def work(case):
    kind, L, p, q, ns = case["kind"], case["L"], case["p"], case["q"], case["nsrc"]
    if kind == "interp2d":
        n = case["nx"] * case["ny"]
        return {"bytes": 8.0 * (4 ** L * p * p + 3 * n), "flops": 2.0 * n * (p * p + p)}
    if kind == "adaptive3d":
        leaves = 300 * (case["sharp"] / 10.0) ** 2  # about what the meshing of these fronts gives
        n, ni, nb = p ** 3, (p - 2) ** 3, 6 * q * q
        return {"bytes": 8.0 * 6 * leaves * n, "flops": _tree_flops(3, 2, ni, n, nb, 1) * leaves / 64.0}
    d = 3 if kind == "dtn3d" else 2
    n, nb = p ** d, 2 * d * q ** (d - 1)
    leaves = (2 ** d) ** L
    size = 16.0 if kind == "iti2d" else 8.0
    terms = 5 if case["terms"] == "full" else d + 1
    bnd = 2 * d * (2 ** L * q) ** (d - 1)
    data = leaves * n * (8.0 * terms + 2 * size * ns) + size * bnd * ns + (size * bnd * bnd if case["top"] else 0)
    if kind == "resolve2d":
        # every stored operator is read once
        ops = leaves * (n * nb + (p - 2) ** 2 * (p - 2) ** 2)
        for lev in range(1, L + 1):
            m = 2 ** (lev - 1) * q
            ops += 4 ** (L - lev) * ((4 * m) ** 2 + 2 * 4 * m * 8 * m)
        return {"bytes": size * (ops + leaves * n * 2 * ns), "flops": 2.0 * ops * ns}
    ni = n if kind == "iti2d" else (p - 2) ** d
    return {"bytes": data, "flops": _tree_flops(d, L, ni, n, nb, ns) * (4.0 if kind == "iti2d" else 1.0)}


def _cost(case):
    """Rough seconds of a pass: keeps drawn cases within the largest listed one."""
    w = work(case)
    if case["kind"] in ("interp2d", "resolve2d"):
        return w["bytes"] / 1e12
    return w["flops"] / (0.5e12 if case["precision"] == "float64" else 5e12)


# ---------------------------------------------------------------------------
# the same discrete problems in 64 bits
# ---------------------------------------------------------------------------


def _cheb(p):
    return np.cos(np.pi * np.arange(p - 1, -1, -1) / (p - 1))


def _interp(src, dst):
    """Barycentric interpolation matrix from the nodes src to dst."""
    w = np.array([1.0 / np.prod(x - np.delete(src, i)) for i, x in enumerate(src)])
    M = np.zeros((len(dst), len(src)))
    for i, t in enumerate(dst):
        d = t - src
        if np.any(d == 0):
            M[i, np.argmin(np.abs(d))] = 1.0
        else:
            M[i] = (w / d) / np.sum(w / d)
    return M


def _diff(x):
    w = np.array([1.0 / np.prod(t - np.delete(x, i)) for i, t in enumerate(x)])
    D = np.array([[0.0 if i == j else (w[j] / w[i]) / (x[i] - x[j]) for j in range(len(x))] for i in range(len(x))])
    return D - np.diag(D.sum(1))


class _Leaf:
    """The leaf grid, its derivative operators, and its boundary maps.

    ``sides[s]`` are the leaf points of side s (2D: S, E, N, W, counter-clockwise; 3D: -x, +x, -y, +y, -z, +z, raster)
    and ``keys`` the places of the boundary nodes, in units of which a leaf is 2q wide."""

    def __init__(self, d, p, q, half, iti_eta=None):
        c, g = _cheb(p), np.polynomial.legendre.leggauss(q)[0]
        D = _diff(c) / half
        ax = np.stack(np.meshgrid(*[np.arange(p)] * d, indexing="ij"), -1).reshape(-1, d)  # (raster point, axis)
        if d == 2:
            ax[:, 1] = p - 1 - ax[:, 1]  # rows run from north to south
        at = {tuple(a): i for i, a in enumerate(ax)}
        m, n = p - 1, p ** d
        if d == 2:
            sides = [[(i, 0) for i in range(p)], [(m, i) for i in range(p)], [(m - i, m) for i in range(p)],
                     [(0, m - i) for i in range(p)]]
            order = [at[s] for side in sides for s in side[:-1]]
            keys = [[(2 * j + 1, 0) for j in range(q)], [(2 * q, 2 * j + 1) for j in range(q)],
                    [(2 * (q - j) - 1, 2 * q) for j in range(q)], [(0, 2 * (q - j) - 1) for j in range(q)]]
            normal = [(1, -1.0), (0, 1.0), (1, 1.0), (0, -1.0)]
            up, down = _interp(g, c), _interp(c, g)
        else:
            sides, keys, normal, order = [], [], [], []
            for a in range(3):
                t = [k for k in range(3) if k != a]
                for e in (0, m):
                    pts = [tuple(x) for x in ax if x[a] == e]
                    sides.append(pts)
                    normal.append((a, 1.0 if e else -1.0))
                    ks = []
                    for i in range(q):
                        for j in range(q):
                            k = [0, 0, 0]
                            k[a], k[t[0]], k[t[1]] = (2 * q if e else 0), 2 * i + 1, 2 * j + 1
                            ks.append(tuple(k))
                    keys.append(ks)
                    order += [at[s] for s in pts if at[s] not in order]
            up, down = np.kron(_interp(g, c), _interp(g, c)), np.kron(_interp(c, g), _interp(c, g))
        inside = [i for i in range(n) if i not in set(order)]
        order = np.array(order + inside)
        self.ncb, self.n = n - len(inside), n
        pos = np.empty(n, dtype=np.int64)
        pos[order] = np.arange(n)
        one = []
        for a in range(d):
            Da = D[::-1, ::-1] if d == 2 and a == 1 else D
            M = np.eye(1)
            for k in range(d):
                M = np.kron(M, Da if k == a else np.eye(p))
            one.append(M[np.ix_(order, order)])
        names = "xyz"
        self.ops = {"I": np.eye(n)}
        for a in range(d):
            self.ops["D_" + names[a]] = one[a]
            for b in range(a, d):
                self.ops["D_" + names[a] + names[b]] = one[a] @ one[b]
        idx = [np.array([pos[at[s]] for s in side]) for side in sides]
        nf = q ** (d - 1)
        self.keys = np.array([k for ks in keys for k in ks])
        N = [sg * one[a][ix] for (a, sg), ix in zip(normal, idx)]
        if iti_eta is None:
            P, count = np.zeros((self.ncb, 2 * d * nf)), np.zeros(self.ncb)
            for s, ix in enumerate(idx):
                P[ix, s * nf:(s + 1) * nf] += up
                count[ix] += 1
            self.P = P / count[:, None]
            self.Q = np.concatenate([down @ Ns for Ns in N])
        else:
            E = np.eye(n)
            self.P = np.kron(np.eye(4), up[:-1]).astype(np.complex128)
            self.G = np.concatenate([(Ns + 1j * iti_eta * E[ix])[:-1] for Ns, ix in zip(N, idx)])
            self.Q = np.concatenate([down @ (Ns - 1j * iti_eta * E[ix]) for Ns, ix in zip(N, idx)])


def _leaf_places(d, L):
    """Grid place of every leaf in tree order."""
    quad = [(0, 0), (1, 0), (1, 1), (0, 1)]
    kids = quad if d == 2 else [(a, b, 1) for a, b in quad] + [(a, b, 0) for a, b in quad]
    at = np.zeros((1, d), dtype=np.int64)
    for _ in range(L):
        at = (2 * at[:, None] + np.array(kids)[None]).reshape(-1, d)
    return at


def _root_order(d, L, q, keys):
    """Positions in ``keys`` of the root's boundary nodes, in the order of the boundary points."""
    where = {tuple(k): i for i, k in enumerate(keys.tolist())}
    w, n = 2 * q * 2 ** L, q * 2 ** L
    if d == 2:
        lst = [(2 * i + 1, 0) for i in range(n)] + [(w, 2 * i + 1) for i in range(n)]
        lst += [(w - 2 * i - 1, w) for i in range(n)] + [(0, w - 2 * i - 1) for i in range(n)]
    else:
        lst = []
        for a in range(3):
            t = [k for k in range(3) if k != a]
            for e in (0, w):
                for pu, pv in _leaf_places(2, L).tolist():
                    for i in range(q):
                        for j in range(q):
                            k = [0, 0, 0]
                            k[a], k[t[0]], k[t[1]] = e, 2 * (pu * q + i) + 1, 2 * (pv * q + j) + 1
                            lst.append(tuple(k))
    return np.array([where[k] for k in lst])


def _solve(A, B):
    return torch.linalg.solve(A, B)


def _exact_pde(case, seed):
    kind, L, p, q = case["kind"], case["L"], case["p"], case["q"]
    d = 3 if kind == "dtn3d" else 2
    iti = kind == "iti2d"
    dev = DEV if torch.cuda.is_available() else "cpu"
    leaf = _Leaf(d, p, q, 1.0 / 2 ** L, float(case["wave"]) if iti else None)
    dt = torch.complex128 if iti else torch.float64
    dom = _domain(case)  # for the places of the points only, which the inputs are functions of
    x, b = torch.as_tensor(dom.interior_points, device=dev), torch.as_tensor(dom.boundary_points, device=dev)
    coeffs, f, g = _inputs(case, seed, x, b)
    del x
    f, g = (t.unsqueeze(-1) if case["nsrc"] == 1 else t for t in (f, g))
    P, Q = torch.as_tensor(leaf.P, device=dev).to(dt), torch.as_tensor(leaf.Q, device=dev).to(dt)
    nl, n, ncb, nb, ns = f.shape[0], leaf.n, leaf.ncb, leaf.Q.shape[0], f.shape[-1]
    Y = torch.empty((nl, n, nb), dtype=dt, device=dev)
    v = torch.zeros((nl, n, ns), dtype=dt, device=dev)
    step = max(1, int(4e8 // (n * n)))
    ops = {k: torch.as_tensor(leaf.ops[k][ncb:], device=dev) for k in coeffs}
    for lo in range(0, nl, step):
        s = slice(lo, min(nl, lo + step))
        A = sum(c[s, ncb:, None] * ops[k] for k, c in coeffs.items()).to(dt)
        m = A.shape[0]
        if iti:
            A = torch.cat([torch.as_tensor(leaf.G, device=dev).expand(m, -1, -1), A], 1)
            scale = 1.0 / A.abs().amax(2, keepdim=True)
            rhs = torch.zeros((m, n, nb + ns), dtype=dt, device=dev)
            rhs[:, :ncb, :nb] = P
            rhs[:, ncb:, nb:] = f[s, ncb:]
            X = _solve(A * scale, rhs * scale)
            Y[s], v[s] = X[..., :nb], X[..., nb:]
        else:
            X = _solve(A[..., ncb:], torch.cat([-A[..., :ncb] @ P, f[s, ncb:]], -1))
            Y[s, :ncb], Y[s, ncb:], v[s, ncb:] = P, X[..., :nb], X[..., nb:]
    at = _leaf_places(d, L)
    flat = np.ravel_multi_index(tuple(at.T), (2 ** L,) * d)
    back = torch.as_tensor(flat, device=dev)
    T = torch.empty((nl, nb, nb), dtype=dt, device=dev)
    h = torch.empty((nl, nb, ns), dtype=dt, device=dev)
    T[back], h[back] = Q @ Y, Q @ v
    grid = [2 ** L] * d
    keys, width, saved = leaf.keys, [2 * q] * d, []
    for _ in range(L):
        for a in range(d):
            T, h = T.reshape(*grid, *T.shape[-2:]), h.reshape(*grid, *h.shape[-2:])
            pick = [tuple(slice(e, None, 2) if k == a else slice(None) for k in range(d)) for e in (0, 1)]
            Ta, Tb, ha, hb = (t[pk].reshape(-1, *t.shape[-2:]) for t, pk in ((T, pick[0]), (T, pick[1]), (h, pick[0]), (h, pick[1])))
            grid[a] //= 2
            kb = keys.copy()
            kb[:, a] += width[a]
            inb = {tuple(k): i for i, k in enumerate(kb.tolist())}
            ia = [i for i, k in enumerate(keys.tolist()) if tuple(k) in inb]
            ib = [inb[tuple(keys[i].tolist())] for i in ia]
            ea, eb = (np.setdiff1d(np.arange(len(keys)), z) for z in (ia, ib))
            ni, na = len(ia), len(ea)
            cross = lambda M, r, c: M[:, r][:, :, c]  # noqa: E731
            Zb = torch.zeros((Ta.shape[0], ni, na), dtype=dt, device=dev)
            Za = torch.zeros((Ta.shape[0], ni, len(eb)), dtype=dt, device=dev)
            if iti:  # x_a = -(outgoing of b), x_b = -(outgoing of a)
                eye = torch.eye(ni, dtype=dt, device=dev).expand(Ta.shape[0], -1, -1)
                K = torch.cat([torch.cat([eye, cross(Tb, ib, ib)], 2), torch.cat([cross(Ta, ia, ia), eye], 2)], 1)
                R = torch.cat([torch.cat([Zb, cross(Tb, ib, eb), hb[:, ib]], 2),
                               torch.cat([cross(Ta, ia, ea), Za, ha[:, ia]], 2)], 1)
            else:
                K = cross(Ta, ia, ia) + cross(Tb, ib, ib)
                R = torch.cat([cross(Ta, ia, ea), cross(Tb, ib, eb), ha[:, ia] + hb[:, ib]], 2)
            X = -_solve(K, R)
            xa, xb = (X[:, :ni], X[:, ni:]) if iti else (X, X)
            Ra, Rb = cross(Ta, ea, ia) @ xa, cross(Tb, eb, ib) @ xb
            ne = na + len(eb)
            Ra[..., :na] += cross(Ta, ea, ea)
            Rb[..., na:ne] += cross(Tb, eb, eb)
            Ra[..., ne:] += ha[:, ea]
            Rb[..., ne:] += hb[:, eb]
            M = torch.cat([Ra, Rb], 1)
            T, h = M[..., :ne].contiguous(), M[..., ne:].contiguous()
            saved.append((a, list(grid), ia, ib, ea, eb, X[..., :ne].contiguous(), X[..., ne:].contiguous()))
            keys = np.concatenate([keys[ea], kb[eb]])
            width[a] *= 2
    order = torch.as_tensor(_root_order(d, L, q, keys), device=dev)
    top = T[0][order][:, order]
    gx = torch.empty((1, len(keys), ns), dtype=dt, device=dev)
    gx[0, order] = g.to(dt)
    del T, h
    while saved:
        a, grid, ia, ib, ea, eb, S, w = saved.pop()
        xi = S @ gx + w
        ni, na = len(ia), len(ea)
        ga = torch.empty((gx.shape[0], ni + na, ns), dtype=dt, device=dev)
        gb = torch.empty((gx.shape[0], ni + len(eb), ns), dtype=dt, device=dev)
        ga[:, ia], gb[:, ib] = (xi[:, :ni], xi[:, ni:]) if iti else (xi, xi)
        ga[:, ea], gb[:, eb] = gx[:, :na], gx[:, na:]
        shape = list(grid)
        shape[a] *= 2
        gx = torch.stack([ga.reshape(*grid, *ga.shape[1:]), gb.reshape(*grid, *gb.shape[1:])], a + 1).reshape(-1, *ga.shape[1:])
    u = Y @ gx[back] + v
    out = {"u": u[..., 0] if ns == 1 else u}
    if case["top"]:
        out["top"] = top
    return out


def _exact_interp(case, seed):
    L, p = case["L"], case["p"]
    dev = DEV if torch.cuda.is_available() else "cpu"
    dom = _domain(case)
    x = torch.as_tensor(dom.interior_points, device=dev)
    s = _bumps(x, np.random.default_rng(int(seed)), 8, 0.3)
    ex, ey = _eval_points(case)
    c, n = _cheb(p), 2 ** L

    def rows(t):
        cell = np.clip(np.floor((t + 1) / 2 * n).astype(np.int64), 0, n - 1)
        loc = (t - (-1 + (2 * cell + 1) / n)) * n
        return cell, torch.as_tensor(_interp(c, loc), device=dev)

    cx, rx = rows(ex)
    cy, ry = rows(ey)
    leaf = _Leaf(2, p, 2, 1.0)
    at = _leaf_places(2, L)
    tree = np.empty((n, n), dtype=np.int64)
    tree[at[:, 0], at[:, 1]] = np.arange(len(at))
    # leaf points as a grid of (x up, y up)
    pos = np.empty((p, p), dtype=np.int64)
    X = dom.interior_points[0]
    ux, uy = np.argsort(np.argsort(_round(X[:, 0]), kind="stable")), np.argsort(np.argsort(_round(X[:, 1]), kind="stable"))
    pos[ux // p, uy // p] = np.arange(leaf.n)
    F = s[:, torch.as_tensor(pos.reshape(-1), device=dev)].reshape(-1, p, p)
    vals = torch.empty((len(ey), len(ex)), dtype=torch.float64, device=dev)
    for j in range(len(ey)):
        blk = F[torch.as_tensor(tree[cx, cy[j]], device=dev)]
        vals[j] = torch.einsum("iab,ia,b->i", blk, rx, ry[j])
    TX, TY = np.meshgrid(ex, ey)
    return {"values": vals.reshape(len(ex), len(ey)), "points": np.stack([TX, TY], 2)}


def _round(t):
    return np.round(t, 10)


def exact(case, seed):
    if case["kind"] == "adaptive3d":
        return None  # a dense system of some 30,000 face unknowns on an uneven tree: minutes
    if case["kind"] == "interp2d":
        return _exact_interp(case, seed)
    return _exact_pde(case, seed)
