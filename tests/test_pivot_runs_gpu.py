"""Fronts around the register tiles of the pivoting kernels: dense symmetric matrices are one root front
of their own order (in registers up to 64, panels of 32 beyond), an arrow of dense blocks gives fronts
with contribution rows. Inertia against numpy's eigenvalues, solutions by their backward error."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _dense(kind, n, rng):
    q = rng.standard_normal((n, n))
    a = 0.5 * (q + q.T)
    if kind == "runs":  # every pivot a plain 1x1 one, both signs
        a += np.diag(np.where(rng.random(n) < 0.5, -1.0, 1.0) * 4.0 * np.sqrt(n))
    elif kind == "pairs":  # zero diagonal: 2x2 pivots
        np.fill_diagonal(a, 0.0)
    elif kind == "mixed":  # runs broken by columns without a usable diagonal
        a += np.diag(np.where(np.arange(n) % 7 == 3, 0.0, 4.0 * np.sqrt(n)))
        a[np.arange(n) % 7 == 3, np.arange(n) % 7 == 3] = 0.0
    return a


def _check(a):
    from hsolve_b200 import Factorization

    w = np.linalg.eigvalsh(a)
    assert np.min(np.abs(w)) > 1e-6 * np.max(np.abs(w)), "a draw whose counts are not defined"
    m = sp.csr_matrix(a)
    f = Factorization(device=0)
    f.analyze(m, None, 1.0, 0.0)
    assert f.factorize(1.0, 0.0)
    got = f.inertia()
    assert (got.neg, got.zero, got.pos) == (int((w < 0).sum()), 0, int((w > 0).sum()))
    c = f.count(1.0, 0.0)
    assert (c.neg, c.zero, c.pos) == (got.neg, got.zero, got.pos)
    assert f.factorize(1.0, 0.0)
    n = a.shape[0]
    b = np.random.default_rng(7).standard_normal((n, 3))
    x = f.solve(b)
    # threshold pivoting with u = 0.01 bounds each multiplier by 100: normwise backward error of a few
    # n eps times that
    eta = np.abs(a @ x - b).max() / (np.abs(a).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max())
    assert eta <= 100 * n * EPS


@pytest.mark.parametrize("kind", ["runs", "pairs", "mixed"])
@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 63, 64, 65, 96, 97, 129, 161, 257])
def test_one_dense_front(kind, n):
    rng = np.random.default_rng(1000 + n)
    _check(_dense(kind, n, rng))


@pytest.mark.parametrize("kind", ["runs", "mixed"])
@pytest.mark.parametrize("n", [1399, 1400, 1457])
def test_pending_pivots_of_large_fronts(kind, n):
    """Fronts of 1,400 rows and more keep 224 pivots pending instead of 128."""
    _check(_dense(kind, n, np.random.default_rng(n)))


@pytest.mark.parametrize("kind", ["runs", "pairs", "mixed"])
@pytest.mark.parametrize("k,c", [(1, 31), (5, 28), (31, 33), (32, 32), (33, 31), (40, 60), (64, 33), (70, 130)])
def test_fronts_with_contribution_rows(kind, k, c):
    """Four dense blocks of order k that couple to a common border of order c."""
    rng = np.random.default_rng(100 * k + c)
    n = 4 * k + c
    a = np.zeros((n, n))
    for t in range(4):
        s = slice(t * k, (t + 1) * k)
        a[s, s] = _dense(kind, k, rng)
        if k == 1:
            a[s, s] = 1.0 - 2.0 * (t % 2)
        e = 0.3 * rng.standard_normal((k, c))
        a[s, 4 * k:] = e
        a[4 * k:, s] = e.T
    a[4 * k:, 4 * k:] = _dense("runs", c, rng)
    _check(a)
