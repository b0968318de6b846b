"""Interface dot products of rows that fill no whole turn of their lanes, and of odd sides: solutions against the global
system, and whole trees against subtrees (whose shorter levels share lanes in other ways) bit for bit."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef
from ellipticforest_gb300 import _lib

pytestmark = pytest.mark.gpu


# row lengths of 4, 8 and 2 sides: shorter than a turn, ending in every part of one, odd and even, two lanes to thirty-two
@pytest.mark.parametrize("n,L", [(3, 2), (5, 4), (7, 3), (9, 5), (11, 3), (14, 3), (15, 4), (17, 4), (18, 5), (23, 2), (33, 2)])
def test_row_ends(lib, n, L):
    from oracle import global_fv as G
    N = n * 2 ** L
    rng = np.random.default_rng(N)
    F, g = rng.standard_normal((N, N)), rng.standard_normal((4, N))
    solver = ef.FiniteVolumeSolver(solver_type=ef.FISHPACK90)
    mesh = ef.Mesh().uniform(L, ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -1.0, 1.0, n, -1.0, 1.0)))
    whole = ef.HPSAlgorithm(mesh, solver)
    whole.buildStage()
    f, r = G.to_leaf_order(F, L, n), g.ravel()
    one, nil = np.ones_like(r), np.zeros_like(r)
    whole.upwards_array(f)
    whole.solve_arrays(one, nil, r)
    u, v = whole.leaf_solution(), G.to_leaf_order(G.solve_poisson_dst(F, *g, -1, 1, -1, 1), L, n)
    assert np.abs(u - v).max() <= 1e-12 * np.abs(v).max()

    cut = L - 1
    parts = [ef.HPSAlgorithm(mesh.subtree(cut, k), solver) for k in range(4 ** cut)]
    top = ef.HPSAlgorithm(mesh, solver)
    for p, fp in zip(parts, np.split(f, len(parts))):
        p.buildStage()
        p.upwards_array(fp)
    top.buildStageTop(cut, [p.root_T() for p in parts])
    top.upwardsStageTop(cut, [p.root_h() for p in parts])
    gs = top.solveStageTop(cut, one, nil, r)
    for k, p in enumerate(parts):
        _lib.check(_lib.load().ef_hps_solve_root_dirichlet(p.handle, _lib.dptr(np.ascontiguousarray(gs[k]))))
    np.testing.assert_array_equal(u, np.concatenate([p.leaf_solution() for p in parts]))
