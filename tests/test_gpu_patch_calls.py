"""Single-patch calls from several threads at once: one at a time works in static device memory and the others
allocate, so every result must be the bits that the same call gives alone."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import ellipticforest_gb300 as ef

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 16, 33, 64])
def test_concurrent_patch_calls(n):
    solver = ef.FiniteVolumeSolver(lambda_function=lambda x, y: -0.7, solver_type=ef.FISHPACK90)

    def call(k):
        rng = np.random.default_rng(100 * n + k)
        grid = ef.FiniteVolumeGrid(n, 0.0, 1.0 + k, n, -1.0, 1.0)
        g, f = rng.standard_normal(4 * n), rng.standard_normal(n * n)
        return solver.solve(grid, g, f), solver.mapD2N(grid, g, f), solver.buildD2N(grid)

    alone = [call(k) for k in range(8)]
    with ThreadPoolExecutor(8) as pool:
        for _ in range(4):
            for got, want in zip(pool.map(call, range(8)), alone):
                for x, y in zip(got, want):
                    np.testing.assert_array_equal(x, y)
