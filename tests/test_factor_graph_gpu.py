"""Repeated factorizations of one object: the launches move into a captured graph after a few uses, which has
to follow the shift, the form (kept factors, counts, null-pivot detection) and a new analysis."""
import numpy as np
import pytest

from helpers import laplacian_2d

pytestmark = pytest.mark.gpu


def test_repeated_factorizations_follow_the_shift_and_the_form():
    from hsolve_b200 import Factorization

    f = Factorization(device=0)
    for nx, ny in ((23, 17), (31, 19)):  # the second analysis replaces the captured work's buffers
        a = laplacian_2d(nx, ny)
        w = np.linalg.eigvalsh(a.toarray())
        rng = np.random.default_rng(nx)
        f.analyze(a, None, 1.0, 0.0)
        for t in range(24):
            # a shift in the middle of one of the wider gaps
            gaps = np.argsort(-np.diff(w))[: w.size // 4]
            g = int(rng.choice(gaps))
            sigma = 0.5 * (w[g] + w[g + 1])
            below = g + 1
            c = f.count(1.0, -sigma, null_pivot_detection=t % 3 != 0)
            assert (c.neg, c.zero, c.pos) == (below, 0, w.size - below)
            assert f.factorize(1.0, -sigma)
            i = f.inertia()
            assert (i.neg, i.zero, i.pos) == (below, 0, w.size - below)
            b = rng.standard_normal((w.size, 1 + t % 3))
            x = f.solve(b)
            r = a @ x - sigma * x - b
            # normwise backward error: multipliers of at most 100, a few roundings per row
            eta = np.abs(r).max() / ((abs(a).sum(axis=1).max() + sigma) * np.abs(x).max() + np.abs(b).max())
            assert eta <= 100 * w.size * np.finfo(float).eps
