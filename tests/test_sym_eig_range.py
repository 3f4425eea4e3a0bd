"""The dense symmetric eigensolver far from unit scale: matrices times powers
of two at which products of three of their entries leave the range of FP64,
and couplings whose squares are near its lower end.  Values within 1e-12 ‖A‖,
vectors parallel to those of the unscaled matrix to 1e-10 (as in
test_sym_eig_edges)."""
import numpy as np
import pytest

from test_lanczos_abi import _check_sym, _sym_eig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 90, 401])
@pytest.mark.parametrize("power", [-400, -350, -101, 101, 350, 400])
def test_powers_of_two(n, power):
    X = np.random.default_rng(n).standard_normal((n, n))
    A = X + X.T
    e0, v0 = _sym_eig(A, n, n)
    e1, v1 = _sym_eig(np.ldexp(A, power), n, n)
    assert np.abs(np.ldexp(e1, -power) - e0).max() <= 1e-12 * np.abs(e0).max()
    assert np.abs(np.ldexp(e1, -power) - np.linalg.eigvalsh(A)).max() <= 1e-12 * np.abs(e0).max()
    sure = np.diff(e0, prepend=-np.inf, append=np.inf)
    sure = np.minimum(sure[:-1], sure[1:]) > 1e-4 * np.abs(e0).max()  # vectors of eps / gap
    assert np.abs(np.abs((v0 * v1).sum(1)) - 1)[sure].max() <= 1e-10


@pytest.mark.parametrize("eps", [1e-150, 1e-154, 1e-155, 1e-158, 1e-161, 1e-163, 1e-300])
def test_tiny_couplings(eps):
    rng = np.random.default_rng(3)
    n = 60
    A = np.zeros((n, n))
    for a, b in ((1, 30), (30, n)):
        X = rng.standard_normal((b - a, b - a))
        A[a:b, a:b] = X + X.T
    A[0, 0] = 0.7
    A[0, 40:44] = A[40:44, 0] = eps
    _check_sym(A, n, n)
