"""The solve operators around the orders of their kernels (32 pivots and less, the 32 and 64 halves of a
super-block of 128, several super-blocks): dense fronts, and dense fronts with contribution rows around
the 64-row tiles and the 256-row chunks, in both factor precisions."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

EPS = {0: np.finfo(np.float64).eps, 1: np.finfo(np.float32).eps}


def _matrix(n, pairs, rng):
    """Symmetric, well conditioned, of both signs; pairs: every third column needs a 2x2 pivot."""
    q = rng.standard_normal((n, n)) / np.sqrt(n)
    a = 0.25 * (q + q.T) + np.diag(np.where(rng.random(n) < 0.5, -2.0, 2.0))
    if pairs:
        for i in range(0, n - 1, 3):
            a[i, i] = a[i + 1, i + 1] = 0.0
            a[i, i + 1] = a[i + 1, i] = 2.0
    return a


def _check(a, precision):
    from hsolve_b200 import Factorization

    m = sp.csr_matrix(a)
    n = a.shape[0]
    f = Factorization(device=0, precision=precision)
    f.analyze(m, None, 1.0, 0.0)
    assert f.factorize(1.0, 0.0)
    for p in (1, 9):
        b = np.random.default_rng(3).standard_normal((n, p))
        x = f.solve(b)
        # multipliers of at most 100 (threshold 0.01), a few roundings per row
        eta = np.abs(a @ x - b).max() / (np.abs(a).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max())
        assert eta <= 100 * n * EPS[precision], (p, eta)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 161, 257, 290])
def test_dense_front(n, pairs, precision):
    _check(_matrix(n, pairs, np.random.default_rng(n)), precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("k,c", [(3, 61), (24, 114), (26, 140), (32, 64), (20, 255), (20, 256), (32, 257), (33, 64), (100, 65), (130, 90),
                                 (160, 300)])
def test_fronts_with_contribution_rows(k, c, precision):
    """Three dense blocks of order k that couple to a common border of order c."""
    rng = np.random.default_rng(k + c)
    n = 3 * k + c
    a = np.zeros((n, n))
    for t in range(3):
        s = slice(t * k, (t + 1) * k)
        a[s, s] = _matrix(k, t == 1, rng)
        e = 0.1 * rng.standard_normal((k, c))
        a[s, 3 * k:] = e
        a[3 * k:, s] = e.T
    a[3 * k:, 3 * k:] = _matrix(c, False, rng) * np.sqrt(1.0 + k)
    _check(a, precision)
