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
