"""Node GEMMs of nodes with equal operators against the same tree with an operator of its own for every node (an
incremental build keeps no classes): operators are stored once, and two nodes go through a tile together, with the same
sums term for term, so the solutions must agree bit for bit."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef
from ellipticforest_gb300._lib import check, load

pytestmark = pytest.mark.gpu


def _codes(row, split):
    s, out = row[1], []
    for kind, K in enumerate((4 * row[1], 2 * row[1], 8 * row[1])):
        if s < 16 or s & (s - 1) or (kind == 1 and s < 32):
            out.append(1)
            continue
        k = 1
        while k < split and (K + 63) // 64 // (2 * k) >= 2:
            k *= 2
        out.append(-k)
    return out


@pytest.mark.parametrize("split", [1, 2, 8])
@pytest.mark.parametrize("kind, B", [("uniform", 5), ("uniform", 40), ("adaptive", 6)])
def test_shared_operators_give_the_same_bits(kind, B, split):
    root = ef.FiniteVolumePatch(ef.FiniteVolumeGrid(16, -1.0, 1.0, 16, -1.0, 1.0))
    mesh = (ef.Mesh().uniform(5, root) if kind == "uniform" else
            ef.Mesh().refineByFunction(lambda x, y: (x - 0.2) ** 2 + (y + 0.3) ** 2 < 0.1, 0.0, 1, 6, root))
    solver = ef.FiniteVolumeSolver(solver_type=ef.FISHPACK90)
    fresh, later = ef.HPSAlgorithm(mesh, solver), ef.HPSAlgorithm(mesh, solver)
    fresh.buildStage()
    assert later.buildStageFrom(fresh) > 0
    rng = np.random.default_rng(B)
    cells = fresh.num_leaves * 256
    F, R = rng.standard_normal((B, cells)), rng.standard_normal((B, 4 * fresh.M))
    A = np.ones((B, 4 * fresh.M))
    got = []
    for h in (fresh, later):
        check(load().ef_hps_set_option(h.handle, b"tensor-cores", 2))
        h.mixed_init(B)
        plan = [(*row[:2], *_codes(row, split)) for row in h.mixed_gemm_plan()]
        h.mixed_set_gemm_plan(plan)
        h.mixed_init(B)
        assert h.mixed_gemm_plan() == plan
        got.append(h.mixed_solve(F, A, R, sweeps=1))
    np.testing.assert_array_equal(got[0], got[1])
