"""Constant-coefficient leaf DtN maps to the last bit: every entry within one unit in the last place of the sum over sine
modes in extended precision.  Entries of opposite sides are many orders below the terms that cancel in them, so a
double-double step that loses its low part shows there."""
import numpy as np
import pytest

import ellipticforest_gb300 as ef

pytestmark = pytest.mark.gpu
LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288419717")


def _exact(n, dx, dy, lam):
    """T (WESN x WESN): with sine modes along the data's side the problem across the patch is one-dimensional."""
    k, j = np.arange(1, n + 1), np.arange(n)
    V = np.sin(PI * LD(1) / (2 * n) * np.outer(k, 2 * j + 1).astype(LD))  # [mode, cell]
    w = np.full(n, LD(2) / n)
    w[-1] /= 2
    out = np.zeros((4, n, 4, n), LD)
    for side in range(4):
        d, g = (dx, dy) if side < 2 else (dy, dx)
        d, g = LD(d), LD(g)
        kappa = (d / g) ** 2 * 4 * np.sin(PI * k.astype(LD) / (2 * n)) ** 2 - LD(lam) * d ** 2
        q = [np.ones(n, LD), 3 + kappa]  # growing solution from the far side, at the cells
        for _ in range(n - 1):
            q.append((2 + kappa) * q[-1] - q[-2])
        q = np.array(q)
        u = 2 * q[:n] / (q[n - 1] + q[n])  # [distance from the far side, mode]
        sol = np.einsum("l,lc,ml,la->cma", w, V, u, V)  # [data cell c, m, cell along]
        near = np.einsum("l,lc,l,la->ca", w, V, (q[n - 1] - q[n]) / (q[n - 1] + q[n]), V)  # u - g at the near cells
        opposite, ends = side ^ 1, ((2, 3) if side < 2 else (0, 1))
        at = np.arange(n) if side & 1 else n - 1 - np.arange(n)  # distance of cell o of a neighbouring side
        s = lambda t: (-2 if t & 1 else 2) / (LD(dx) if t < 2 else LD(dy))
        out[side, :, side, :] = s(side) * near.T
        out[opposite, :, side, :] = s(opposite) * sol[:, 0, :].T
        for t, e in zip(ends, (0, n - 1)):
            out[t, :, side, :] = s(t) * sol[:, at, e].T
    return out.reshape(4 * n, 4 * n)


@pytest.mark.parametrize("n,box,lam", [(2, (0, 1, 0, 1), 0.0), (5, (-1, 1, 0, 0.5), -3.0), (8, (0, 1, 0, 1), 9.0),
                                       (16, (-1, 1, -1, 1), 0.0), (17, (0, 2, 0, 1), -1.0), (32, (0, 1, 0, 1), 0.0)])
def test_entries_to_the_last_bit(lib, n, box, lam):
    if np.finfo(LD).nmant < 100:
        pytest.skip("extended precision of this machine is no reference for the cancelling entries")
    T = ef.FiniteVolumeSolver(lambda_function=lambda x, y: lam, solver_type=ef.FISHPACK90).buildD2N(
        ef.FiniteVolumeGrid(n, box[0], box[1], n, box[2], box[3]))
    E = _exact(n, (box[1] - box[0]) / n, (box[3] - box[2]) / n, lam)
    # one rounding of the scaled sum and one of the spacing; the sum itself carries some 2^-100 of its terms
    assert np.all(np.abs(T.astype(LD) - E) <= 2.0 ** -52 * np.abs(E) + 2.0 ** -96 * np.abs(E).max())
