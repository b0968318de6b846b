"""The build's digit products by themselves, against exact integers: the error of every entry within the stated bound, for
digits without a pattern, rows and columns graded over many powers of two, and digits that make the left-out pairs as
large as they get."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def product(lib, tmp_path_factory):
    from ellipticforest_gb300 import build
    so = tmp_path_factory.mktemp("digits") / "digit_product.so"
    cmd = [build.nvcc(), "-shared", *build.ARCH, *build.COMMON, *build.CU_FLAGS, str(ROOT / "tests/cpp/digit_product.cu"), "-o", str(so)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    fn = C.CDLL(str(so)).digit_product

    def run(A, B):
        A, B = np.ascontiguousarray(A), np.ascontiguousarray(B)
        out = np.empty((A.shape[0], B.shape[1]))
        p = lambda x: x.ctypes.data_as(C.c_void_p)
        assert fn(p(A), p(B), p(out), A.shape[0], B.shape[1], A.shape[1]) == 0
        return out
    return run


def _ints(X, unit):
    """Entries as exact integers in units of 2^-unit."""
    out = np.empty(X.shape, object)
    for i, x in np.ndenumerate(X):
        a, b = float(x).as_integer_ratio()
        out[i] = (a << unit) // b
    return out


def _check(product, A, B):
    K = A.shape[1]
    got = _ints(product(A, B), 2148)
    a, b = _ints(A, 1074), _ints(B, 1074)
    exact = a.dot(b)
    scale = np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None, :]
    assert np.all(np.abs(got - exact) * 2 ** 62 <= 33 * K * scale + np.abs(exact) * 2 ** 9)
    return np.abs(got - exact), K * scale


# one tile and several, ends of tiles and of k blocks
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (33, 31, 65), (128, 32, 128), (130, 70, 200)])
@pytest.mark.parametrize("spread", [0, 30, 300])
def test_error_within_the_bound(product, M, N, K, spread):
    rng = np.random.default_rng(M + K + spread)
    graded = lambda *s: rng.standard_normal(s) * 2.0 ** rng.integers(-spread, spread + 1, s)
    _check(product, graded(M, K), graded(K, N))


@pytest.mark.parametrize("K", [64, 192])
def test_largest_left_out_pairs(product, K):
    # 0.5 sets a row's (column's) scale so that it is twice its largest entry; the others have the digits 0, 0, -128 .. -128
    tail = -sum(128 * 256.0 ** (7 - i) for i in range(2, 8)) * 2.0 ** -62
    A, B = np.full((40, K), tail), np.full((K, 40), tail)
    A[:, 0], B[-1, :] = 0.5, 0.5
    err, unit = _check(product, A, B)
    # five of the seven pairs of weight 8 here: 20 of the bound's 33
    assert np.all(err * 2 ** 62 >= 19 * (K - 2) * unit // K)


def test_rows_that_are_not_finite(product):
    rng = np.random.default_rng(0)
    A, B = rng.standard_normal((40, 70)), rng.standard_normal((70, 40))
    want = product(A, B)
    A[3, 5], A[7, 0], B[1, 9] = np.inf, np.nan, -np.inf
    got = product(A, B)
    bad = np.zeros((40, 40), bool)
    bad[[3, 7]] = True
    bad[:, 9] = True
    assert np.isnan(got[bad]).all()
    np.testing.assert_array_equal(got[~bad], want[~bad])
