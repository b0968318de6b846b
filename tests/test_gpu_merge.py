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
