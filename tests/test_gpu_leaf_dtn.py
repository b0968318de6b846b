"""Leaf DtN maps on the GPU against the oracle's."""
import numpy as np
import pytest

from oracle import hps_oracle as O

pytestmark = pytest.mark.gpu


# the smallest and odd sides, cells 60 times longer than wide, and lambda on either side of half the smallest
# eigenvalue of the patch (19.74 on a unit square in the limit; below the double-double sums, above the LU)
@pytest.mark.parametrize("n,box,lam", [(2, (0, 1, 0, 1), 0.0), (3, (0, 1, 0, 2), -2.0), (5, (0, 1, 0, 60), 0.0),
                                       (9, (0, 60, 0, 1), -1.0), (17, (0, 1, 0, 1), 9.0), (17, (0, 1, 0, 1), 10.5),
                                       (33, (-1, 1, 0, 1), 0.0)])
def test_constant_coefficient_map_matches_oracle(lib, n, box, lam):
    import ellipticforest_gb300 as ef
    T = ef.FiniteVolumeSolver(lambda_function=lambda x, y: lam, solver_type=ef.FISHPACK90).buildD2N(
        ef.FiniteVolumeGrid(n, box[0], box[1], n, box[2], box[3]))
    To = O.FiniteVolumeSolver(solver_type=O.FISHPACK90, lambda_function=lambda x, y: lam).buildD2N(
        O.FiniteVolumeGrid(n, box[0], box[1], n, box[2], box[3]))
    assert np.abs(T - To).max() <= 1e-12 * np.abs(To).max()


# FivePointStencil leaves: every block width of the column kernel (8, 16, 24, 32) full and ragged, the row
# kernel beyond 32; maps, solutions and fluxes of one patch and the maps of a whole tree
@pytest.mark.parametrize("n", [2, 3, 8, 11, 16, 17, 23, 24, 25, 31, 32, 34])
def test_variable_coefficient_leaves_match_oracle(lib, n):
    import ellipticforest_gb300 as ef
    co = dict(alpha_function=lambda x, y: 1.0 + 0.2 * x * y, beta_function=lambda x, y: 1.0 + 0.5 * np.sin(3 * x) * np.cos(2 * y),
              lambda_function=lambda x, y: -1.0 - x * x)
    solver, oracle = ef.FiniteVolumeSolver(**co), O.FiniteVolumeSolver(**co)
    rng = np.random.default_rng(n)
    g, f = rng.standard_normal(4 * n), rng.standard_normal(n * n)
    gg, og = ef.FiniteVolumeGrid(n, -1, 1, n, 0, 1), O.FiniteVolumeGrid(n, -1, 1, n, 0, 1)
    rel = lambda a, b: np.abs(a - b).max() / np.abs(b).max()
    assert rel(solver.buildD2N(gg), oracle.buildD2N(og)) <= 1e-12
    assert rel(solver.solve(gg, g, f), oracle.solve(og, g, f)) <= 1e-12
    assert rel(solver.mapD2N(gg, g, f), oracle.mapD2N(og, g, f)) <= 1e-12
    # one leaf, so the tree's root map is the leaf's, from the kernels that build all leaves' maps at once
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(0, ef.FiniteVolumePatch(gg)), solver)
    hps.buildStage()
    assert rel(hps.root_T(), oracle.buildD2N(og)) <= 1e-12
