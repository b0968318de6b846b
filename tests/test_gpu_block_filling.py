"""The requests that fill a block of the mixed solver up to a multiple of four are zero requests: their solutions are zeros."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef

pytestmark = pytest.mark.gpu


class _Buffer:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


@pytest.mark.parametrize("bmax,held", [(7, 8), (23, 24)])
def test_filling_requests_are_zero(lib, bmax, held):
    import torch
    patch = ef.FiniteVolumePatch(ef.FiniteVolumeGrid(16, -1.0, 1.0, 16, -1.0, 1.0))
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(2, patch), ef.FiniteVolumeSolver(solver_type=ef.FISHPACK90))
    hps.buildStage()
    hps.mixed_init(bmax)
    rng = np.random.default_rng(bmax)
    cells = hps.num_leaves * 256
    f, r = rng.standard_normal((bmax, cells)), rng.standard_normal((bmax, 4 * hps.M))
    u = hps.mixed_solve(f, np.ones_like(r), r, 1)
    places = torch.as_tensor(_Buffer(hps.mixed_buffers()[3], (held, cells)), device="cuda").cpu().numpy()
    np.testing.assert_array_equal(places[:bmax], u)
    assert np.all(places[bmax:] == 0.0)
