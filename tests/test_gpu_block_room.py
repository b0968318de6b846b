"""Device memory of block solvers: room beyond the block's requests only where a full block is filled up."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef

pytestmark = pytest.mark.gpu


def test_room_grows_with_the_requests(lib):
    patch = ef.FiniteVolumePatch(ef.FiniteVolumeGrid(16, -1.0, 1.0, 16, -1.0, 1.0))
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(5, patch), ef.FiniteVolumeSolver(solver_type=ef.FISHPACK90))
    hps.buildStage()
    got = {}
    for b in (4, 5, 6, 7, 8, 13, 16):
        srv = ef.Server([hps], bmax=b, lanes=1)
        got[b] = srv.device_bytes()
        del srv
    per = (got[8] - got[4]) / 4
    # requests held: 7 is filled up to 8, the others are more than a sixth short of a multiple of four
    for b, held in ((5, 5), (6, 6), (7, 8), (13, 13), (16, 16)):
        assert abs(got[b] - got[4] - (held - 4) * per) <= 0.05 * per
