"""The work that users of the HPS solver have it do, as cases that can be timed.

A case is one pass through the public entry points: a single-patch solve, a right-hand side on a
resident factored tree, a factorisation followed by a solve, or a block of right-hand sides through
the mixed-precision block solver.  Loads are sums of Gaussian bumps, root data are a few Fourier modes
per side, variable coefficients are smooth and positive: the data of the repository's benchmark, drawn
from the case's seed.

A tree is ``uniform`` (level L, n x n cells per leaf patch, so N = n 2^L cells per side) or ``adaptive``
(refined where |sin x + sin y| exceeds ``cut`` on [-10, 10]^2, up to level L).  ``leaf`` names the leaf
solver: the constant-coefficient one or the FivePointStencil one with variable beta.
"""
import math

import numpy as np
import torch

import ellipticforest_gb300 as ef

DEVICE = "cuda"


def _case(kind, leaf="constant", tree="uniform", L=0, n=16, box=1.0, lam=0.0, bc="dirichlet", cut=1.2, B=1, sweeps=0):
    return {"kind": kind, "leaf": leaf, "tree": tree, "L": L, "n": n, "box": box, "lam": lam, "bc": bc, "cut": cut,
            "B": B, "sweeps": sweeps}


def listed():
    def named(name, *a, **k):
        return {"name": name, **_case(*a, **k)}
    return [
        # one patch of the plug-in interface, host arrays in and out: the smallest call there is
        named("patch_16", "patch", box=10.0),
        # a right-hand side on a small resident tree: launch latency (the single-process example, 64 leaves)
        named("solve_L3_16", "solve", L=3, box=10.0),
        # a right-hand side on the largest uniform tree (2048^2 cells)
        named("solve_L7_16", "solve", L=7),
        # factor and solve a small tree, as a program does that solves once per mesh
        named("build_L4_16", "build", L=4),
        # factor and solve at 1024^2 cells
        named("build_L6_16", "build", L=6),
        # factor and solve at 2048^2 cells: the largest
        named("build_L7_16", "build", L=7),
        # flux data on two sides (the heat-conduction driver): the general dense root solve joins in; ragged patches
        named("build_flux_L5_10", "build", L=5, n=10, lam=-1.0, bc="flux"),
        # factor and solve on an adaptive tree with uneven level jumps (coarsening inside the merges)
        named("build_adaptive_16", "build", tree="adaptive", L=7, box=10.0),
        # variable coefficients: every leaf and every merge has an operator of its own
        named("build_variable_L5_32", "build", leaf="variable", L=5, n=32, lam=-1.0),
        # a block of requests on the largest tree, mixed precision with one refinement sweep: throughput
        named("block_L7_16", "block", L=7, B=32, sweeps=1),
        # a block of requests on the adaptive tree (two sweeps), a block size that fills no tile
        named("block_adaptive_16", "block", tree="adaptive", L=7, box=10.0, B=23, sweeps=2),
        # a block of requests with variable coefficients
        named("block_variable_L5_32", "block", leaf="variable", L=5, n=32, lam=-1.0, B=16, sweeps=1),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)) ) - 0.5)))


def draw(rng):
    kind = rng.choice(["patch", "solve", "solve", "build", "build", "build", "block", "block"])
    box, lam = rng.choice([1.0, 10.0, 0.3]), rng.choice([0.0, 0.0, -1.0, -3.5])
    if kind == "patch":
        return _case(kind, n=_log(rng, 4, 64), box=box, lam=lam)
    leaf = rng.choice(["constant", "constant", "variable"])
    if leaf == "constant" and rng.random() < 0.3:
        n = rng.choice([8, 12, 16])
        return _case(kind, tree="adaptive", L=rng.randint(4, 6), n=n, box=10.0, cut=round(rng.uniform(1.0, 1.6), 3),
                     **(dict(B=_log(rng, 1, 40), sweeps=2) if kind == "block" else {}))
    most = 480 if leaf == "variable" else 1024
    cells = rng.uniform(math.log(32), math.log(most))
    L = rng.randint(1, 6 if leaf == "constant" else 5)
    n = min(32, max(4, round(math.exp(cells) / 2 ** L)))
    if kind == "block":
        n = max(4, n // 4 * 4)
        return _case(kind, leaf=leaf, L=L, n=n, box=1.0, lam=lam, B=_log(rng, 1, 64), sweeps=1)
    bc = "flux" if leaf == "constant" and n * 2 ** L <= 400 and rng.random() < 0.3 else "dirichlet"
    return _case(kind, leaf=leaf, L=L, n=n, box=box, lam=-1.0 if bc == "flux" else lam, bc=bc)


# -- the seeded data of a case ---------------------------------------------------------------------
def _dev():
    return DEVICE if torch.cuda.is_available() else "cpu"


def _beta(seed):
    p, q = np.random.default_rng((seed, 7)).uniform(-0.5, 0.5, 2)
    return lambda x, y: 1.0 + 0.5 * np.sin(np.pi * (x + p)) * np.cos(np.pi * (y + q))


def _load(seed, b, X, Y):
    """Load of request b at points of [-1, 1]^2 (tensors)."""
    rng = np.random.default_rng((seed, 11, b))
    f = torch.zeros_like(X)
    for amp, cx, cy, w in zip(rng.uniform(-1, 1, 8), *rng.uniform(-1, 1, (2, 8)), rng.uniform(0.05, 0.3, 8)):
        f += amp * torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / w ** 2)
    return f


def _root(seed, b, M):
    """Root data of request b: [4, M], sides W, E, S, N."""
    co = np.random.default_rng((seed, 13, b)).standard_normal((4, 6))
    t = (np.arange(M) + 0.5) / M
    return torch.from_numpy(co @ np.sin(np.pi * np.arange(1, 7)[:, None] * t)).to(_dev())


def _ab(case, M):
    """Root operator a u + b du/dn on the 4M root faces."""
    a, b = torch.ones(4, M, dtype=torch.float64, device=_dev()), torch.zeros(4, M, dtype=torch.float64, device=_dev())
    if case["bc"] == "flux":
        a[2:], b[2:] = 0.0, 1.0
    return a, b


def _zorder(L):
    z = np.arange(4 ** L)
    ix, iy = np.zeros_like(z), np.zeros_like(z)
    for k in range(L):
        ix |= ((z >> (2 * k)) & 1) << k
        iy |= ((z >> (2 * k + 1)) & 1) << k
    return torch.from_numpy(ix * 2 ** L + iy).to(_dev())


def _to_leaves(U, L, n):
    """A global N x N cell array (x outer) in leaf order, cell j + i n of each leaf."""
    return U.reshape(2 ** L, n, 2 ** L, n).permute(0, 2, 1, 3).reshape(4 ** L, n * n)[_zorder(L)].reshape(-1)


def _unit_grid(N):
    t = (torch.arange(N, dtype=torch.float64, device=_dev()) + 0.5) * (2.0 / N) - 1.0
    return t[:, None].expand(N, N), t[None, :].expand(N, N)


# -- a user's program ------------------------------------------------------------------------------
def _mesh(case):
    n, r = case["n"], case["box"]
    root = ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -r, r, n, -r, r))
    if case["tree"] == "uniform":
        return ef.Mesh().uniform(case["L"], root)
    cut = case["cut"]
    return ef.Mesh().refineByFunction(lambda x, y: abs(math.sin(x) + math.sin(y)) > cut, cut, 0, case["L"], root)


def _solver(case, seed):
    lam = case["lam"]
    if case["leaf"] == "variable":
        return ef.FiniteVolumeSolver(alpha_function=lambda x, y: 1.0 + 0.0 * x, beta_function=_beta(seed),
                                     lambda_function=lambda x, y: lam + 0.0 * x, solver_type=ef.FivePointStencil)
    return ef.FiniteVolumeSolver(lambda_function=lambda x, y: lam, solver_type=ef.FISHPACK90)


def _loads(case, seed, mesh):
    if case["tree"] == "uniform":
        X, Y = _unit_grid(case["n"] * 2 ** case["L"])
        for b in range(case["B"]):
            yield _to_leaves(_load(seed, b, X, Y), case["L"], case["n"])
    else:
        X, Y = (torch.from_numpy(v / case["box"]).to(_dev()) for v in mesh.cell_centres())
        for b in range(case["B"]):
            yield _load(seed, b, X, Y)


class _Buffer:
    """A device buffer of the library as a tensor."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _tensor(ptr, shape, owner):
    return torch.as_tensor(_Buffer(ptr, shape, owner), device=DEVICE)


def prepare(case, seed):
    if case["kind"] == "patch":
        n, r = case["n"], case["box"]
        rng = np.random.default_rng((seed, 3))
        g, f = rng.standard_normal(4 * n), rng.standard_normal(n * n)
        return {"kind": "patch", "solver": _solver(case, seed), "g": g, "f": f,
                "grid": ef.FiniteVolumeGrid(n, -r, r, n, -r, r)}
    mesh = _mesh(case)
    hps = ef.HPSAlgorithm(mesh, _solver(case, seed))
    hps.setupStage()
    cells = hps.num_leaves * hps.n * hps.n
    if case["kind"] != "build":
        hps.buildStage()
    if case["kind"] == "block":
        B = case["B"]
        hps.mixed_init(B)
        f, a, r, u = hps.mixed_buffers()
        F, A, R = _tensor(f, (B, cells), hps), _tensor(a, (B, 4 * hps.M), hps), _tensor(r, (B, 4 * hps.M), hps)
        A.fill_(1.0)
        for b, load in enumerate(_loads(case, seed, mesh)):
            F[b] = load
            R[b] = _root(seed, b, hps.M).reshape(-1)
        return {"kind": "block", "hps": hps, "B": B, "sweeps": case["sweeps"], "u": _tensor(u, (B, cells), hps)}
    f = next(_loads(case, seed, mesh)).contiguous()
    a, b = _ab(case, hps.M)
    return {"kind": case["kind"], "hps": hps, "f": f, "a": a, "b": b, "r": _root(seed, 0, hps.M).contiguous(),
            "dirichlet": case["bc"] == "dirichlet", "u": _tensor(hps.device_buffers()[1], (cells,), hps)}


def run(state):
    if state["kind"] == "patch":
        s, grid, g, f = state["solver"], state["grid"], state["g"], state["f"]
        return {"u": s.solve(grid, g, f), "h": s.mapD2N(grid, g, f)}
    hps = state["hps"]
    if state["kind"] == "block":
        hps.mixed_solve_async(state["B"], state["sweeps"])
        return state["u"]
    if state["kind"] == "build":
        hps.buildStage()
    hps.load_device_async(*(state[k].data_ptr() for k in ("f", "a", "b", "r")))
    hps.solve_device_async(state["dirichlet"])
    return state["u"]


# -- what a pass cannot do without -----------------------------------------------------------------
def _merges(case):
    """(number of nodes, distinct operators, interface points m = 4 s) per level of a uniform tree.  With
    constant coefficients all nodes of a level have the same operator; with variable ones each has its own."""
    for lvl in range(case["L"]):
        cnt = 4 ** lvl
        yield cnt, (1 if case["leaf"] == "constant" else cnt), 4 * case["n"] * 2 ** (case["L"] - 1 - lvl)


def work(case):
    n, B = case["n"], case["B"]
    if case["kind"] == "patch":
        return {"bytes": 2 * 8 * (2 * n * n + 4 * n) + 8 * 4 * n, "flops": 2 * 8 * n ** 3}
    if case["tree"] == "adaptive":
        # the root merge of an adaptive tree has the leaf patch's size at least: loads and solutions bound it
        cells = _mesh(case).num_leaves() * n * n
        return {"bytes": B * 2 * 8 * cells, "flops": B * cells * 8 * n}
    cells, M = (n * 2 ** case["L"]) ** 2, n * 2 ** case["L"]
    leaf = 6 * n if case["leaf"] == "constant" else 4 * n  # multiply-adds per cell of a leaf solve
    nbytes, flops = B * (2 * 8 * cells + 4 * 8 * M), B * 2 * leaf * cells
    for cnt, own, m in _merges(case):
        entries = 4 * m * m  # S (m x 2m), X^-1 (m x m), compact H (2m x m/2)
        if case["kind"] == "build":
            flops += own * (2 / 3 + 6 + 4) * m ** 3  # LU of X, X^-1 [S I], T += H S
            nbytes += own * 8 * (entries + 4 * m * m)
        else:
            nbytes += own * (4 if case["kind"] == "block" else 8) * entries
        flops += B * cnt * 2 * entries * (1 + case["sweeps"])
    if case["bc"] == "flux":
        flops += 2 / 3 * (4 * M) ** 3 if case["kind"] == "build" else 2 * (4 * M) ** 2
    return {"bytes": nbytes, "flops": flops}


# -- the same in 64 bits ---------------------------------------------------------------------------
def _basis(N, d, kind, dev):
    """Orthonormal eigenvectors (rows) and eigenvalues of the 1-D second difference with Dirichlet ('s') or flux ('c') ends."""
    k = torch.arange(N, dtype=torch.float64, device=dev) + (1.0 if kind == "s" else 0.0)
    i = torch.arange(N, dtype=torch.float64, device=dev) + 0.5
    arg = math.pi / N * torch.outer(k, i)
    V = (torch.sin(arg) if kind == "s" else torch.cos(arg)) * math.sqrt(2.0 / N)
    V[-1 if kind == "s" else 0] /= math.sqrt(2.0)
    return V, -(4.0 / d ** 2) * torch.sin(math.pi * k / (2 * N)) ** 2


def _constant_solve(F, g, d, lam, bc):
    """u with the 5-point operator + lam = F and root data g (W, E, S, N) of the whole N x N grid."""
    N = F.shape[0]
    F = F.clone()
    F[0] -= 2 / d ** 2 * g[0]
    F[-1] -= 2 / d ** 2 * g[1]
    if bc == "flux":
        F[:, 0] += g[2] / d
        F[:, -1] -= g[3] / d
    else:
        F[:, 0] -= 2 / d ** 2 * g[2]
        F[:, -1] -= 2 / d ** 2 * g[3]
    Vx, ex = _basis(N, d, "s", F.device)
    Vy, ey = _basis(N, d, "c" if bc == "flux" else "s", F.device)
    return Vx.T @ ((Vx @ F @ Vy.T) / (ex[:, None] + ey[None, :] + lam)) @ Vy


def _variable_solve(F, g, d, lam, beta, box):
    """u with div(beta grad u) + lam u = F: conjugate gradients preconditioned with the constant operator."""
    N = F.shape[0]
    t = -box + (np.arange(N) + 0.5) * d
    X, Y = np.meshgrid(t, t, indexing="ij")
    faces = lambda v: torch.from_numpy(v).to(F.device)
    bW, bE = faces(beta(X - d / 2, Y)), faces(beta(X + d / 2, Y))
    bS, bN = faces(beta(X, Y - d / 2)), faces(beta(X, Y + d / 2))

    def apply(u, g=None):
        gW, gE, gS, gN = (torch.zeros(N, dtype=u.dtype, device=u.device),) * 4 if g is None else g
        west, east, south, north = (torch.empty_like(u) for _ in range(4))
        west[1:], west[0] = u[:-1] - u[1:], 2 * (gW - u[0])
        east[:-1], east[-1] = u[1:] - u[:-1], 2 * (gE - u[-1])
        south[:, 1:], south[:, 0] = u[:, :-1] - u[:, 1:], 2 * (gS - u[:, 0])
        north[:, :-1], north[:, -1] = u[:, 1:] - u[:, :-1], 2 * (gN - u[:, -1])
        return ((bW * west + bE * east) + (bS * south + bN * north)) / d ** 2 + lam * u

    zero = torch.zeros(4, N, dtype=F.dtype, device=F.device)
    precondition = lambda r: _constant_solve(r, zero, d, lam, "dirichlet")
    u = torch.zeros_like(F)
    for _ in range(3):  # restarts: the residual anew, differences first
        r = F - apply(u, g)
        z = precondition(r)
        p, rz = z.clone(), float((r * z).sum())
        first = abs(rz)
        while first > 0 and abs(rz) > 1e-24 * first:
            q = apply(p)
            step = rz / float((p * q).sum())
            u += step * p
            r -= step * q
            z = precondition(r)
            rz, old = float((r * z).sum()), rz
            p = z + (rz / old) * p
    return u


def exact(case, seed):
    n, r = case["n"], case["box"]
    if case["kind"] == "patch":
        rng = np.random.default_rng((seed, 3))
        g, f = rng.standard_normal(4 * n), rng.standard_normal(n * n)
        g, f = torch.from_numpy(g).reshape(4, n), torch.from_numpy(f).reshape(n, n)
        d = 2 * r / n
        u = _constant_solve(f, g, d, case["lam"], "dirichlet")
        h = torch.stack([u[0] - g[0], g[1] - u[-1], u[:, 0] - g[2], g[3] - u[:, -1]]) * (2 / d)
        return {"u": u.reshape(-1).numpy(), "h": h.reshape(-1).numpy()}
    if case["tree"] == "adaptive":
        return None
    N = n * 2 ** case["L"]
    d = 2 * r / N
    X, Y = _unit_grid(N)
    out = []
    for b in range(case["B"]):
        F, g = _load(seed, b, X, Y), _root(seed, b, N)
        if case["leaf"] == "variable":
            u = _variable_solve(F, g, d, case["lam"], _beta(seed), r)
        else:
            u = _constant_solve(F, g, d, case["lam"], case["bc"])
        out.append(_to_leaves(u, case["L"], n))
    return torch.stack(out) if case["kind"] == "block" else out[0]
