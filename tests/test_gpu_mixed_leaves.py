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
