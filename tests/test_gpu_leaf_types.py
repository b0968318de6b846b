"""Leaf DtN maps of trees with several leaf types: a type's map depends on the type alone, so that an incremental build
and a split into subtrees, whose trees have other types beside it, give the same bits as one whole tree."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef
from ellipticforest_gb300 import _lib

pytestmark = pytest.mark.gpu


def _mesh(refine, lo, hi, n, r):
    patch = ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -r, r, n, -r, r))
    return ef.Mesh().refineByFunction(refine, 0.0, lo, hi, patch)


def _data(hps, n):
    rng = np.random.default_rng(n)
    return rng.standard_normal(hps.num_leaves * n * n), rng.standard_normal(4 * hps.M)


# lambda = 15 lies above half the smallest eigenvalue of the leaves of level 2 (side 1, 2 pi^2 = 19.7 in the limit) and
# below it on level 3; odd n too
@pytest.mark.parametrize("n,lam", [(5, 0.0), (7, -1.0), (8, 15.0), (5, 15.0)])
def test_incremental_build_and_subtrees_equal_a_fresh_build(lib, n, lam):
    solver = ef.FiniteVolumeSolver(lambda_function=lambda x, y: lam, solver_type=ef.FISHPACK90)
    mesh = _mesh(lambda x, y: x < -0.25, 2, 3, n, 2.0)
    fresh = ef.HPSAlgorithm(mesh, solver)
    fresh.buildStage()
    f, r = _data(fresh, n)
    one, nil = np.ones(4 * fresh.M), np.zeros(4 * fresh.M)
    fresh.upwards_array(f)
    fresh.solve_arrays(one, nil, r)

    # from a tree that has leaves of one level only
    for refine in (lambda x, y: True, lambda x, y: False):
        old = ef.HPSAlgorithm(_mesh(refine, 2, 3, n, 2.0), solver)
        old.buildStage()
        inc = ef.HPSAlgorithm(mesh, solver)
        assert inc.buildStageFrom(old) > 0
        np.testing.assert_array_equal(fresh.root_T(), inc.root_T())

    cut = 1
    parts = [ef.HPSAlgorithm(mesh.subtree(cut, k), solver) for k in range(4)]
    top = ef.HPSAlgorithm(mesh, solver)
    for p, fp in zip(parts, np.split(f, np.cumsum([p.num_leaves * n * n for p in parts])[:-1])):
        p.buildStage()
        p.upwards_array(fp)
    top.buildStageTop(cut, [p.root_T() for p in parts])
    top.upwardsStageTop(cut, [p.root_h() for p in parts])
    g = top.solveStageTop(cut, one, nil, r)
    for k, p in enumerate(parts):
        _lib.check(_lib.load().ef_hps_solve_root_dirichlet(p.handle, _lib.dptr(np.ascontiguousarray(g[k]))))
    np.testing.assert_array_equal(fresh.leaf_solution(), np.concatenate([p.leaf_solution() for p in parts]))
