"""Merges that block elimination gives up go through the pivoted LU, those of a level together; the levels below them are
not merged again."""
import numpy as np
import pytest
import scipy.sparse.linalg as spla

import ellipticforest_gb300 as ef

pytestmark = pytest.mark.gpu


def _checker(m, k):
    """1 and 10^k on squares of side 1 / m; the faces of cells whose centres lie beside an edge see one of the two"""
    return lambda x, y: np.where((np.floor(x * m + 1e-9) + np.floor(y * m + 1e-9)) % 2 == 0, 1.0, 10.0 ** k) + 0.0 * y


# coefficients that jump inside the leaves (most nodes of some levels given up), and indefinite operators (few); 9: a level
# of odd children keeps the LU beside them
@pytest.mark.parametrize("n,L,beta,lam", [(10, 3, _checker(7, 6), 0.0), (16, 3, _checker(7, 3), 0.0), (10, 3, None, 2000.0),
                                          (9, 3, None, 2000.0), (16, 3, None, 500.0)])
def test_rejected_merges(lib, n, L, beta, lam):
    from oracle import global_fv as G
    N = n * 2 ** L
    F = np.random.default_rng(N).standard_normal((N, N))
    if beta is None:
        solver = ef.FiniteVolumeSolver(lambda_function=lambda x, y: lam, solver_type=ef.FISHPACK90)
    else:
        solver = ef.FiniteVolumeSolver(beta_function=beta, lambda_function=lambda x, y: lam)
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(L, ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -1.0, 1.0, n, -1.0, 1.0))), solver)
    u = []
    for k in range(3):  # eager, captured, replayed with the merges given up again
        hps.profile_enable(k == 0)
        hps.buildStage()
        if k == 0:
            p = hps.profile()
            assert 1 <= p["getrf"]["calls"] <= L
        hps.upwards_array(G.to_leaf_order(F, L, n))
        z = np.zeros(4 * N)
        hps.solve_arrays(z + 1, z, z)
        u.append(hps.leaf_solution())
    np.testing.assert_array_equal(u[0], u[1])
    np.testing.assert_array_equal(u[0], u[2])
    A = G.assemble(N, N, -1, 1, -1, 1, beta=beta, lam=lambda X, Y: lam + 0 * X)[0].tocsc()
    lu = spla.splu(A)
    v = G.to_leaf_order(lu.solve(F.ravel()).reshape(N, N), L, n)
    inv = spla.LinearOperator(A.shape, matvec=lu.solve, rmatvec=lambda x: lu.solve(x, "T"), dtype=float)
    # relative error of a backward stable solve: a few eps times the condition number
    assert np.abs(u[0] - v).max() <= 64 * 2.0 ** -53 * spla.onenormest(A) * spla.onenormest(inv) * np.abs(v).max()
