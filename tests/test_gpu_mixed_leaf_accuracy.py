"""Accuracy of one FP32 solve of a variable-coefficient leaf: no worse than block substitution with its products formed one
after the other (T = q - L y, then L_jj^-1 T) in FP32, as an average over a block's requests."""
import numpy as np
import pytest
import scipy.sparse.linalg as spla

import ellipticforest_gb300 as ef
from oracle import global_fv as G

pytestmark = pytest.mark.gpu


def _substitute(A, n, Q):
    """Block LU of A in FP64 (blocks of n rows), its block rows in FP32, Q solved with them."""
    blk = lambda i, j: A[i * n:(i + 1) * n, j * n:(j + 1) * n]
    f32 = lambda x: np.asarray(x, np.float32)
    Linv, Lsub, Uinv, Usup = [], [], [], []
    for j in range(n):
        D = blk(j, j).copy()
        if j:
            Lsub.append(blk(j, j - 1) @ Uinv[-1])
            D -= Lsub[-1] @ Usup[-1]
        L, U = np.eye(n), D
        for k in range(n):
            L[k + 1:, k] = U[k + 1:, k] / U[k, k]
            U[k + 1:] -= np.outer(L[k + 1:, k], U[k])
        Linv.append(np.linalg.inv(L))
        Uinv.append(np.linalg.inv(np.triu(U)))
        if j < n - 1:
            Usup.append(Linv[-1] @ blk(j, j + 1))

    def product(M, x):  # one chain of FP32 multiply-adds per entry
        s = np.zeros_like(x)
        for k in range(n):
            s = f32(s.astype(np.float64) + M[:, k:k + 1].astype(np.float64) * x[k:k + 1].astype(np.float64))
        return s
    Linv, Lsub, Uinv, Usup = ([f32(m) for m in ms] for ms in (Linv, Lsub, Uinv, Usup))
    y = [f32(Q[j * n:(j + 1) * n]) for j in range(n)]
    for j in range(n):
        y[j] = product(Linv[j], y[j] - product(Lsub[j - 1], y[j - 1]) if j else y[j])
    for j in range(n - 1, -1, -1):
        y[j] = product(Uinv[j], y[j] - product(Usup[j], y[j + 1]) if j < n - 1 else y[j])
    return np.concatenate(y).astype(np.float64)


@pytest.mark.parametrize("n", [16, 32])
def test_leaf_solve_error(lib, n):
    B = 64
    beta = lambda x, y: 1.0 + 0.5 * np.sin(np.pi * x + 0.3) * np.cos(np.pi * y - 0.2)
    solver = ef.FiniteVolumeSolver(beta_function=beta, lambda_function=lambda x, y: -1.0 + 0.0 * x)
    hps = ef.HPSAlgorithm(ef.Mesh().uniform(0, ef.FiniteVolumePatch(ef.FiniteVolumeGrid(n, -1.0, 1.0, n, -1.0, 1.0))), solver)
    hps.buildStage()
    hps.mixed_init(B)
    F = np.random.default_rng(n).standard_normal((B, n * n)).astype(np.float32).astype(np.float64)
    r = np.zeros((B, 4 * n))
    u = hps.mixed_solve(F, r + 1.0, r, 0)
    A = G.assemble(n, n, -1, 1, -1, 1, beta=beta, lam=lambda X, Y: -1.0 + 0 * X)[0]
    exact = spla.splu(A.tocsc()).solve(F.T)
    mean = lambda x: np.mean(np.linalg.norm(x - exact, axis=0) / np.linalg.norm(exact, axis=0))
    # (averages of 64 requests: a tenth is several times their spread)
    assert mean(u.T) <= 1.1 * mean(_substitute(A.toarray(), n, F.T))
