"""The workspace of builds and general root solves: a refused request leaves the one there is in place, the kept memory is
counted, and a limit gives it back."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef
from ellipticforest_gb300 import _lib

pytestmark = pytest.mark.gpu


def _tree():
    patch = ef.FiniteVolumePatch(ef.FiniteVolumeGrid(8, -1.0, 1.0, 8, -1.0, 1.0))
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(5, patch), ef.FiniteVolumeSolver(lambda_function=lambda x, y: -1.0,
                                                                            solver_type=ef.FISHPACK90))
    return hps, hps.device_bytes


def _limit(hps, mb):
    _lib.check(_lib.load().ef_hps_set_option(hps.handle, b"workspace-limit-mb", mb))


# the merges' largest level (side 128) takes 20 MB, the root operator (1024 rows) 25.5 MB
@pytest.mark.parametrize("limit", [0, 23])
def test_refused_root_scratch_leaves_the_merges_theirs(lib, limit):
    hps, arena = _tree()
    _limit(hps, limit)
    hps.buildStage()
    T = hps.root_T()
    kept = hps.device_bytes - arena
    assert 20 << 20 <= kept <= 23 << 20
    rng = np.random.default_rng(0)
    f, r = rng.standard_normal(hps.num_leaves * 64), rng.standard_normal(4 * hps.M)
    hps.upwards_array(f)
    hps.solve_arrays(np.ones_like(r), 0.5 * np.ones_like(r), r)
    u = hps.leaf_solution()
    assert (hps.device_bytes - arena > kept) == (limit == 0)
    for _ in range(3):  # eager, captured, replayed
        hps.buildStage()
        np.testing.assert_array_equal(hps.root_T(), T)
    # the root operator inverted and factored: a few eps times its condition number apart (diagonal 1 + 0.5 |T|)
    other, _ = _tree()
    _limit(other, 23 if limit == 0 else 0)
    other.buildStage()
    other.upwards_array(f)
    other.solve_arrays(np.ones_like(r), 0.5 * np.ones_like(r), r)
    assert np.abs(other.leaf_solution() - u).max() <= 1e-11 * np.abs(u).max()


def test_limit_gives_back_and_merges_by_lu(lib):
    hps, arena = _tree()
    hps.buildStage()
    T = hps.root_T()
    _limit(hps, 1)
    assert hps.device_bytes == arena
    for _ in range(3):
        hps.buildStage()
    by_lu = hps.root_T()
    assert hps.device_bytes <= arena + (1 << 20)
    assert np.abs(by_lu - T).max() <= 1e-12 * np.abs(T).max()
    _limit(hps, 0)
    hps.buildStage()
    np.testing.assert_array_equal(hps.root_T(), T)
