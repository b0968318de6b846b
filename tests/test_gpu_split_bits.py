"""A right-hand side on a whole tree against the same tree as a top part and subtrees, bit for bit: the long levels of
the whole tree and the short ones of a subtree share out their dot products in different ways, and few leaves are spread
over more blocks (16 x 16 ones by a kernel of their own), but every sum is added in one order."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef
from ellipticforest_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L, n, cut", [(6, 16, 2), (6, 10, 3), (5, 13, 2), (5, 32, 2), (5, 7, 1), (4, 33, 2), (3, 64, 2)])
def test_subtrees_equal_the_whole_tree(L, n, cut):
    solver = ef.FiniteVolumeSolver(solver_type=ef.FISHPACK90)
    mesh = ef.Mesh().uniform(L, ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -1.0, 1.0, n, -1.0, 1.0)))
    whole = ef.HPSAlgorithm(mesh, solver)
    whole.buildStage()
    rng = np.random.default_rng(L * 100 + n)
    f, r = rng.standard_normal(whole.num_leaves * n * n), rng.standard_normal(4 * whole.M)
    one, nil = np.ones(4 * whole.M), np.zeros(4 * whole.M)
    whole.upwards_array(f)
    whole.solve_arrays(one, nil, r)

    parts = [ef.HPSAlgorithm(mesh.subtree(cut, k), solver) for k in range(4 ** cut)]
    top = ef.HPSAlgorithm(mesh, solver)
    for p, fp in zip(parts, np.split(f, len(parts))):
        p.buildStage()
        p.upwards_array(fp)
    top.buildStageTop(cut, [p.root_T() for p in parts])
    top.upwardsStageTop(cut, [p.root_h() for p in parts])
    g = top.solveStageTop(cut, one, nil, r)
    for k, p in enumerate(parts):
        _lib.check(_lib.load().ef_hps_solve_root_dirichlet(p.handle, _lib.dptr(np.ascontiguousarray(g[k]))))
    np.testing.assert_array_equal(whole.leaf_solution(), np.concatenate([p.leaf_solution() for p in parts]))
