"""Copies of the caller's large pageable arrays in pinned stripes: sizes
around the smallest striped one and around a stripe's chunks, arrays that
start anywhere, every host-array entry point, and two handles in two threads."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIN = (8 << 20) // 8  # values in the smallest striped array
# alpha is 1 up to two sums over the same products in different orders: at most
# 2,000 serial additions each way, 2,000 * 2 * 1.1e-16
RTOL = 4.4e-13


def _diagonal(n, seed):
    from xsolver_b200 import CSRMatrix

    rng = np.random.default_rng(seed)
    d = 2.0 ** rng.integers(-3, 4, n)  # powers of two: one step solves, but for alpha's rounding
    return CSRMatrix(n, np.arange(n + 1), np.arange(n), d)


def _at(a, offset):
    """a's values in an array that starts offset values into its allocation."""
    out = np.empty(a.size + offset, a.dtype)[offset:]
    out[:] = a
    return out


def _check(n, offset, seed):
    from xsolver_b200.api import Solver

    A = _diagonal(n, seed)
    b = _at(np.random.default_rng(seed + 1).standard_normal(n), offset)
    S = Solver(A).ksp_settype("pcg").ksp_setoption(1e-10, 5).pc_settype("jacobi")
    x = S.solve(b)
    assert np.allclose(x, b / A.val, rtol=RTOL, atol=0)
    g = _at(np.random.default_rng(seed + 2).standard_normal(n), offset)
    db, dA = S.adjoint(g)
    assert np.allclose(db, g / A.val, rtol=RTOL, atol=0)
    assert np.allclose(dA, -db * x, rtol=RTOL, atol=0)
    v = _at(A.val[::-1].copy(), offset)
    S.mat_update(v)
    assert np.allclose(S.solve(b), b / v, rtol=RTOL, atol=0)
    S.close()


@pytest.mark.parametrize("n", [MIN - 1, MIN, MIN + 1, 8 * (1 << 18) + 511, 3 * MIN + 77777])
def test_solve_update_adjoint(cuda, n):
    for offset in (0, 1):
        _check(n, offset, n % 97)


@pytest.mark.parametrize("k", [2, 3])
def test_batch(cuda, k):
    from xsolver_b200.api import Solver

    n = MIN // 2 + 1001
    A = _diagonal(n, k)
    B = np.random.default_rng(k).standard_normal((k, n))
    S = Solver(A).ksp_settype("pcg").ksp_setoption(1e-10, 5).pc_settype("jacobi")
    X = S.solve_batch(B)
    assert np.allclose(X, B / A.val, rtol=RTOL, atol=0)
    G = np.random.default_rng(k + 9).standard_normal((k, n))
    DB, DA = S.adjoint_batch(X, G)
    assert np.allclose(DB, G / A.val, rtol=RTOL, atol=0)
    assert np.allclose(DA, -DB * X, rtol=RTOL, atol=0)


def test_two_handles_in_two_threads(cuda):
    failed = []

    def run(seed):
        try:
            for _ in range(3):
                _check(MIN + 4321, seed % 2, seed)
        except BaseException as e:  # noqa: BLE001
            failed.append(e)

    th = [threading.Thread(target=run, args=(s,)) for s in (1, 2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not failed
