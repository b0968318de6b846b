"""Inputs loaded from device memory at any 8-byte alignment, all or some of them, and the general root solve at sizes
around its blocks of 32 and 128 unknowns."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef

pytestmark = pytest.mark.gpu


def _tree(n, L):
    root = ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -1.0, 1.0, n, -1.0, 1.0))
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(L, root), ef.FiniteVolumeSolver(
        lambda_function=lambda x, y: -1.0, solver_type=ef.FISHPACK90))
    hps.buildStage()
    return hps


@pytest.mark.parametrize("n, L", [(2, 1), (5, 2), (8, 3), (13, 2), (16, 3)])
def test_loaded_inputs_at_any_alignment(n, L):
    import torch
    hps = _tree(n, L)
    rng = np.random.default_rng(n)
    f, r = rng.standard_normal(hps.num_leaves * n * n), rng.standard_normal(4 * hps.M)
    one, nil = np.ones(4 * hps.M), np.zeros(4 * hps.M)

    def at(x, off):  # a device copy of x at `off` doubles past an allocation's start
        t = torch.zeros(x.size + 8, dtype=torch.float64, device="cuda")
        t[off:off + x.size] = torch.from_numpy(x)
        return t[off:]

    got = []
    for offs in ((0, 0, 0, 0), (1, 2, 3, 1), (3, 1, 0, 2)):
        t = [at(x, o) for x, o in zip((f, one, nil, r), offs)]
        torch.cuda.synchronize()
        hps.load_device_async(*(x.data_ptr() for x in t))
        hps.solve_device_async(True)
        hps.synchronize()
        got.append(hps.leaf_solution())
    # only the load again, halved: root data stay
    half = at(0.5 * f, 1)
    torch.cuda.synchronize()
    hps.load_device_async(half.data_ptr())
    hps.solve_device_async(True)
    hps.synchronize()
    got.append(hps.leaf_solution())
    want = []
    for load in (f, 0.5 * f):
        hps.upwards_array(load)
        hps.solve_arrays(one, nil, r)
        want.append(hps.leaf_solution())
    for k, u in enumerate(got):
        np.testing.assert_array_equal(u, want[k == 3])


@pytest.mark.parametrize("n, L", [(2, 1), (4, 1), (5, 1), (7, 1), (9, 1), (8, 2), (10, 2), (16, 2), (33, 1), (10, 4)])
def test_general_root_solve_returns_the_dirichlet_data(n, L):
    hps = _tree(n, L)
    rng = np.random.default_rng(n + L)
    m = 4 * hps.M
    f, g = rng.standard_normal(hps.num_leaves * n * n), rng.standard_normal(m)
    hps.upwards_array(f)
    hps.solve_arrays(np.ones(m), np.zeros(m), g)
    want = hps.leaf_solution()
    a, b = rng.uniform(0.5, 1.5, m), rng.uniform(0.1, 0.2, m)
    T, h = hps.root_T(), hps.root_h()
    hps.solve_arrays(a, b, a * g + b * (T @ g + h))
    got = hps.leaf_solution()
    # root data of a backward stable solve, and the solution by them (bounded by its boundary values for lambda <= 0)
    Z = np.diag(a) + b[:, None] * T
    scale = np.abs(g).max() + np.abs(b[:, None] * T).sum(1).max() * 2.0 * np.abs(g).max()
    tol = 64 * 2.0 ** -53 * np.linalg.cond(Z) * scale
    assert np.abs(got - want).max() <= tol
