"""Leaf solves of the mixed block solver with variable coefficients, against the plain FP64 solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# leaf sides with idle lanes and full ones; blocks below, at and past the eight requests of a warp and the
# sixteen of a thread block
@pytest.mark.parametrize("n,L,B", [(4, 2, 1), (8, 2, 9), (12, 1, 16), (20, 2, 17), (32, 1, 8), (32, 2, 37)])
def test_variable_coefficient_blocks_match_plain(lib, n, L, B):
    import ellipticforest_gb300 as ef
    solver = ef.FiniteVolumeSolver(beta_function=lambda x, y: 1.0 + 0.5 * np.sin(3 * x) * np.cos(2 * y),
                                   lambda_function=lambda x, y: -1.0 - x * x)
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(L, ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -1, 1, n, -1, 1))), solver)
    hps.buildStage()
    hps.mixed_init(B)
    rng = np.random.default_rng(n)
    f, r = rng.standard_normal((B, hps.num_leaves * n * n)), rng.standard_normal((B, 4 * hps.M))
    u = hps.mixed_solve(f, np.ones_like(r), r, 2)
    for b in {0, B // 2, B - 1}:
        hps.upwards_array(f[b])
        hps.solve_arrays(np.ones(4 * hps.M), np.zeros(4 * hps.M), r[b])
        v = hps.leaf_solution()
        assert np.abs(u[b] - v).max() <= 1e-10 * np.abs(v).max()


# full blocks that are filled up to a multiple of four (6, 7, 11) or not (5, 13), and a smaller block of the same
# solver, whose neighbours' rows must stay as they were
@pytest.mark.parametrize("bmax", [5, 6, 7, 11, 13])
def test_blocks_of_any_size_match_single_requests(lib, bmax):
    import ellipticforest_gb300 as ef
    patch = ef.FiniteVolumePatch(ef.FiniteVolumeGrid(8, -10, 10, 8, -10, 10))
    mesh = ef.Mesh().refineByFunction(lambda x, y: abs(np.sin(x) + np.sin(y)) > 1.2, 1.2, 0, 4, patch)
    hps = ef.HPSAlgorithm(mesh, ef.FiniteVolumeSolver(solver_type=ef.FISHPACK90))
    hps.buildStage()
    rng = np.random.default_rng(bmax)
    f, r = rng.standard_normal((bmax, hps.num_leaves * 64)), rng.standard_normal((bmax, 4 * hps.M))
    hps.mixed_init(1)
    one = np.concatenate([hps.mixed_solve(f[b], np.ones_like(r[b]), r[b], 1) for b in range(bmax)])
    hps.mixed_init(bmax)
    u = hps.mixed_solve(f, np.ones_like(r), r, 1)
    assert np.array_equal(u, one)
    assert np.array_equal(hps.mixed_solve(f[:bmax - 1], np.ones_like(r[1:]), r[:bmax - 1], 1), one[:bmax - 1])
    assert np.isfinite(hps.mixed_residuals(2)[:, :bmax - 1]).all()
