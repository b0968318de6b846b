"""A general root solve that fails while it inverts a new operator keeps nothing of the one before: the next solve with the
old operator inverts it again."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef
from ellipticforest_gb300 import _lib

pytestmark = pytest.mark.gpu


def test_failed_root_inverse_is_not_taken_for_the_old_one(lib):
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(3, ef.FiniteVolumePatch(ef.FiniteVolumeGrid(8, -1.0, 1.0, 8, -1.0, 1.0))),
                          ef.FiniteVolumeSolver(lambda_function=lambda x, y: -1.0, solver_type=ef.FISHPACK90))
    hps.buildStage()
    rng = np.random.default_rng(0)
    f, r = rng.standard_normal(hps.num_leaves * 64), rng.standard_normal(4 * hps.M)
    one = np.ones_like(r)
    hps.upwards_array(f)

    def solve(b):
        hps.solve_arrays(one, b * one, r)
        return hps.leaf_solution()
    u = solve(0.5)
    _lib.check(_lib.load().ef_hps_set_option(hps.handle, b"inject-merge-error", 1))
    with pytest.raises(_lib.EFError) as e:
        solve(0.25)
    assert e.value.code == _lib.EF_ERR_CUDA and "did not complete" in str(e.value)
    _lib.check(_lib.load().ef_hps_set_option(hps.handle, b"inject-merge-error", 0))
    np.testing.assert_array_equal(u, solve(0.5))
    assert not np.array_equal(u, solve(0.25))
