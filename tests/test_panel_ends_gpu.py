"""2x2 pivots at the ends of panels: fronts of 2x2 blocks with contribution rows whose last panel is narrower than
32 and ends with a pair, or whose panels of 32 split a pair, in both factor precisions; and fronts around the
order from which more pivots stay pending."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

EPS = {0: np.finfo(np.float64).eps, 1: np.finfo(np.float32).eps}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [2047, 2048, 2113])
def test_pending_pivots_around_the_larger_fronts(n, precision):
    """Fronts of 2,048 rows and more keep 224 pivots pending instead of 128: plain pivots of both signs, broken by
    columns that need a 2x2 pivot, in a matrix of known eigenvalue signs (diagonally dominant blocks)."""
    from hsolve_b200 import Factorization

    rng = np.random.default_rng(n)
    q = rng.standard_normal((n, n)) / n
    a = q + q.T + np.diag(np.where(np.arange(n) % 3 == 0, -3.0, 3.0))  # |q + q^T| has norm below 1
    neg = int((np.arange(n) % 3 == 0).sum())
    for i in range(40, n - 1, 97):  # a pair of eigenvalues +-3 in the place of the two diagonal entries
        neg += 1 - int(a[i, i] < 0) - int(a[i + 1, i + 1] < 0)
        a[i, i] = a[i + 1, i + 1] = 0.0
        a[i, i + 1] = a[i + 1, i] = 3.0
    f = Factorization(device=0, precision=precision)
    f.analyze(sp.csr_matrix(a), None, 1.0, 0.0, pivot_order=np.arange(1, n + 1))
    assert f.factorize(1.0, 0.0)
    i = f.inertia()
    assert (i.neg, i.zero, i.pos) == (neg, 0, n - neg)
    b = rng.standard_normal((n, 2))
    x = f.solve(b)
    eta = np.abs(a @ x - b).max() / (np.abs(a).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max())
    assert eta <= 100 * n * EPS[precision]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("first", [0, 1])  # 1: a plain pivot first, so that the panels of 32 split pairs
@pytest.mark.parametrize("k", [66, 74, 95, 98, 130])
@pytest.mark.parametrize("c", [3, 40, 600])
def test_pairs_at_the_ends(k, c, first, precision):
    from hsolve_b200 import Factorization

    rng = np.random.default_rng(k + 7 * c + first)
    n = 2 * k + c
    a = np.zeros((n, n))
    for t in range(2):
        s = slice(t * k, (t + 1) * k)
        q = 0.05 * rng.standard_normal((k, k)) / np.sqrt(k)
        d = q + q.T
        np.fill_diagonal(d, 0.0)
        d[0, 0] = 2.0 * first
        for i in range(first, k - 1, 2):
            d[i, i + 1] = d[i + 1, i] = 2.0
        if (k - first) % 2:
            d[k - 1, k - 1] = 2.0
        a[s, s] = d
        e = 0.1 * rng.standard_normal((k, c)) / np.sqrt(k)
        a[s, 2 * k:] = e
        a[2 * k:, s] = e.T
    q = 0.1 * rng.standard_normal((c, c)) / np.sqrt(c)
    a[2 * k:, 2 * k:] = q + q.T + 3.0 * np.eye(c)
    w = np.linalg.eigvalsh(a)
    m = sp.csr_matrix(a)
    f = Factorization(device=0, precision=precision)
    f.analyze(m, None, 1.0, 0.0, pivot_order=np.arange(1, n + 1))  # the blocks' own order: pairs stay together
    assert f.factorize(1.0, 0.0)
    i = f.inertia()
    assert (i.neg, i.zero, i.pos) == (int((w < 0).sum()), 0, int((w > 0).sum()))
    assert i.two_by_two >= k // 4
    b = rng.standard_normal((n, 3))
    x = f.solve(b)
    # multipliers of at most 100 (threshold 0.01), a few roundings per row
    eta = np.abs(a @ x - b).max() / (np.abs(a).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max())
    assert eta <= 100 * n * EPS[precision]
