"""A wait that gives up while a build redoes its rejected merges: the build reports it, the handle is not built, and the
next build does not inherit it.  The error word is set as the kernel would set it; nothing on the GPU waits."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef
from ellipticforest_gb300 import _lib

pytestmark = pytest.mark.gpu
N = 16


def _eig(cells):
    """Lowest eigenvalue of the 1-D second difference on `cells` cells of width 1 / N."""
    return 4.0 * N ** 2 * np.sin(np.pi / (2 * cells)) ** 2


def _mesh(L, n):
    return ef.Mesh().uniform(L, ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -1.0, 1.0, n, -1.0, 1.0)))


# lambda cancels the lowest eigenvalue of the left half: the block that the elimination starts with is singular
RESONANCE = _eig(N) + _eig(2 * N)


def _refused(hps, build):
    _lib.check(_lib.load().ef_hps_set_option(hps.handle, b"inject-merge-error", 1))
    with pytest.raises(_lib.EFError) as e:
        build()
    assert e.value.code == _lib.EF_ERR_CUDA and "did not complete" in str(e.value)
    u = np.zeros(hps.num_leaves * hps.n * hps.n)
    assert _lib.load().ef_hps_upwards(hps.handle, _lib.dptr(u)) == _lib.EF_ERR_STATE
    _lib.check(_lib.load().ef_hps_set_option(hps.handle, b"inject-merge-error", 0))
    try:  # (a constant lambda makes the whole operator singular too)
        build()
    except _lib.EFError as e:
        assert e.code == _lib.EF_ERR_SINGULAR


def test_build(lib):
    lam = lambda x, y: np.where(x < 0, RESONANCE, -1.0) + 0.0 * y
    hps = ef.HPSAlgorithm(_mesh(1, N), ef.FiniteVolumeSolver(beta_function=lambda x, y: 1.0 + 0.0 * x, lambda_function=lam))
    hps.buildStage()
    f, r = np.random.default_rng(0).standard_normal(4 * N * N), np.zeros(8 * N)

    def solve():
        hps.upwards_array(f)
        hps.solve_arrays(np.ones_like(r), r, r)
        return hps.leaf_solution()
    u = solve()
    _refused(hps, hps.buildStage)
    np.testing.assert_array_equal(u, solve())


def test_incremental_build(lib):
    solver = ef.FiniteVolumeSolver(lambda_function=lambda x, y: RESONANCE, solver_type=ef.FISHPACK90)
    old = ef.HPSAlgorithm(_mesh(0, N), solver)
    old.buildStage()
    hps = ef.HPSAlgorithm(_mesh(1, N), solver)
    _refused(hps, lambda: hps.buildStageFrom(old))


def test_top_of_a_split_tree(lib):
    solver = ef.FiniteVolumeSolver(lambda_function=lambda x, y: RESONANCE, solver_type=ef.FISHPACK90)
    mesh = _mesh(2, N // 2)
    parts = [ef.HPSAlgorithm(mesh.subtree(1, k), solver) for k in range(4)]
    for p in parts:
        p.buildStage()
    top = ef.HPSAlgorithm(mesh, solver)
    _refused(top, lambda: top.buildStageTop(1, [p.root_T() for p in parts]))
