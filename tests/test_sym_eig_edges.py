"""The dense symmetric eigensolver at the edges of its blocks: sizes around
multiples of eight reflectors and of a warp, rows that are already reduced
(no reflector), blocks that do not couple, and matrices scaled by powers of
two (the reduction does not normalise its reflectors).  Bounds as in
test_lanczos_abi: values within 1e-12 ‖A‖, residuals within 1e-11 ‖A‖, vectors
orthonormal to 1e-10 (and parallel to those of the scaled matrix)."""
import numpy as np
import pytest

from test_lanczos_abi import _check_sym, _sym_eig


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 8, 9, 10, 11, 18, 19, 31, 33, 127, 129, 255, 257, 639])
def test_sizes(n):
    X = np.random.default_rng(n).standard_normal((n, n))
    _check_sym(X + X.T, n, n)
    _check_sym(X + X.T, 3, 2)


@pytest.mark.gpu
def test_rows_without_a_reflector():
    rng = np.random.default_rng(7)
    n = 75
    T = np.diag(rng.standard_normal(n)) + np.diag(rng.standard_normal(n - 1), 1)
    _check_sym(T + T.T, n, n)  # tridiagonal already
    A = np.zeros((n, n))  # two dense blocks around a diagonal stretch
    for a, b in ((0, 30), (41, n)):
        X = rng.standard_normal((b - a, b - a))
        A[a:b, a:b] = X + X.T
    A[np.arange(30, 41), np.arange(30, 41)] = rng.standard_normal(11)
    _check_sym(A, n, n)
    P = rng.permutation(n)
    _check_sym(A[np.ix_(P, P)], n, n)


@pytest.mark.gpu
@pytest.mark.parametrize("power", [-120, 120])
def test_scaling(power):
    X = np.random.default_rng(11).standard_normal((90, 90))
    A = X + X.T
    e0, v0 = _sym_eig(A, 20, 20)
    e1, v1 = _sym_eig(A * 2.0 ** power, 20, 20)
    assert np.allclose(e1, e0 * 2.0 ** power, rtol=1e-11, atol=1e-12 * np.abs(e0).max() * 2.0 ** power)
    assert np.abs(np.abs((v0 * v1).sum(1)) - 1).max() <= 1e-10
