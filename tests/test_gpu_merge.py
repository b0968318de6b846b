"""Merges of the build on the GPU: nodes with equal operators merge once, with the same result as
when each merges for itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ef(lib):
    import ellipticforest_gb300
    return ellipticforest_gb300


# box 0.3: midpoint halving gives neighbouring leaves spacings that differ in the last bit, so a level
# has several distinct merges; the adaptive tree has coarsened children of several sizes
@pytest.mark.parametrize("box,n,L,adaptive", [((-1, 1, -1, 1), 8, 3, False), ((-0.3, 0.3, -0.3, 0.7), 6, 4, False),
                                              ((-10, 10, -10, 10), 8, 5, True), ((-0.3, 10, -0.7, 10), 8, 5, True)])
def test_equal_merges_match_separate_ones(ef, box, n, L, adaptive):
    patch = lambda: ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, box[0], box[1], n, box[2], box[3]))
    solver = ef.FiniteVolumeSolver(solver_type=ef.FISHPACK90)
    if adaptive:
        mesh = ef.Mesh().refineByFunction(lambda x, y: abs(np.sin(x) + np.sin(y)) > 1.2, 1.2, 0, L, patch())
    else:
        mesh = ef.Mesh().uniform(L, patch())
    once = ef.HPSAlgorithm(mesh, solver)
    once.buildStage()
    # an incremental build that finds nothing to reuse merges every node for itself
    old = ef.HPSAlgorithm(ef.Mesh().uniform(1, patch()), solver)
    old.buildStage()
    each = ef.HPSAlgorithm(mesh, solver)
    assert each.buildStageFrom(old) == 0
    assert np.array_equal(once.root_T(), each.root_T())
    f = np.random.default_rng(L).standard_normal(once.num_leaves * n * n)
    r = np.random.default_rng(n).standard_normal(4 * once.M)
    u = []
    for h in (once, each):
        h.upwards_array(f)
        h.solve_arrays(np.ones_like(r), np.zeros_like(r), r)
        u.append(h.leaf_solution())
    assert np.array_equal(*u)


def _solve(ef, n, L, lam=0.0, beta=None, seed=0):
    """Random loads and root data on [-1,1]^2: the build's solution and the global system's."""
    from oracle import global_fv as G
    N = n * 2 ** L
    rng = np.random.default_rng(seed)
    F, g = rng.standard_normal((N, N)), rng.standard_normal((4, N))
    root = ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -1.0, 1.0, n, -1.0, 1.0))
    kind = ef.FISHPACK90 if beta is None else ef.FivePointStencil
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(L, root), ef.FiniteVolumeSolver(
        beta_function=beta, lambda_function=lambda x, y: lam, solver_type=kind))
    hps.buildStage()
    hps.upwards_array(G.to_leaf_order(F, L, n))
    r = g.ravel()
    hps.solve_arrays(np.ones_like(r), np.zeros_like(r), r)
    if beta is None:
        u = G.solve_poisson_dst(F, *g, -1, 1, -1, 1, lam=lam)
    else:
        side = lambda x, y: g[0 if x[0] == x[-1] == -1 else 1 if x[0] == x[-1] == 1 else 2 if y[0] == -1 else 3]
        u = G.solve_dirichlet(N, N, -1, 1, -1, 1, lambda X, Y: F, side, beta=beta,
                              lam=lambda X, Y: lam + 0 * X)[0]
    return hps.leaf_solution(), G.to_leaf_order(u, L, n)


# child sides s = n 2^k from the smallest that takes the tensor-core products (8) over sides that fill no
# block of 32, 64 or 128 (10, 20, 40; 12 .. 48; 18 .. 72) to several tiles each way; odd s keeps the LU
@pytest.mark.parametrize("n,L", [(8, 1), (16, 1), (9, 2), (10, 3), (12, 3), (18, 3), (20, 3), (33, 2), (16, 5)])
@pytest.mark.parametrize("variable", [False, True])
def test_build_sizes_match_global_solve(ef, n, L, variable):
    beta = (lambda x, y: 1.0 + 0.5 * np.sin(np.pi * x) * np.cos(np.pi * y)) if variable else None
    if variable and n * 2 ** L > 200:
        pytest.skip("sparse LU of the global system")
    u, v = _solve(ef, n, L, lam=-1.0 if variable else 0.0, beta=beta)
    assert np.abs(u - v).max() <= 1e-12 * np.abs(v).max()


@pytest.mark.parametrize("n", [16, 24])
def test_merge_with_a_singular_leading_block_takes_the_pivoted_lu(ef, n):
    # lambda cancels the lowest eigenvalue of the two patches of the left half: the block that the
    # elimination of the interface matrix starts with is singular, the whole matrix is not
    from oracle import global_fv as G
    e = lambda N: 4.0 * n ** 2 * np.sin(np.pi / (2 * N)) ** 2
    lam = lambda x, y: np.where(x < 0, e(n) + e(2 * n), -1.0) + 0.0 * y
    one = lambda x, y: 1.0 + 0.0 * x
    root = ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -1.0, 1.0, n, -1.0, 1.0))
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(1, root), ef.FiniteVolumeSolver(beta_function=one, lambda_function=lam))
    hps.buildStage()
    F = np.random.default_rng(n).standard_normal((2 * n, 2 * n))
    hps.upwards_array(G.to_leaf_order(F, 1, n))
    hps.solve_arrays(np.ones(8 * n), np.zeros(8 * n), np.zeros(8 * n))
    A = G.assemble(2 * n, 2 * n, -1, 1, -1, 1, beta=one, lam=lam)[0].toarray()
    v = G.to_leaf_order(np.linalg.solve(A, F.ravel()).reshape(2 * n, 2 * n), 1, n)
    # relative error of a backward stable solve: a few eps times the condition number
    assert np.abs(hps.leaf_solution() - v).max() <= 64 * 2.0 ** -53 * np.linalg.cond(A) * np.abs(v).max()
