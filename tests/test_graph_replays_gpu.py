"""Which factorizations are replayed from a captured graph, and that the replayed ones are right: every form of one
object (kept factors, counts, with and without null-pivot detection) in both factor precisions, the orders around
the largest that is captured, objects in two threads, and a session's concurrent shifts."""
import threading

import numpy as np
import pytest

from helpers import laplacian_1d, laplacian_2d

pytestmark = pytest.mark.gpu

USES = 8  # a form's first captured use
SOLVE_GRAPHS = 64  # most captured solves of an object
LARGEST = 65536  # largest order whose factorizations are captured


def _gaps(w, count):
    """Shifts in the middle of the widest gaps of the ascending spectrum w, and the eigenvalues below them."""
    g = np.sort(np.argsort(-np.diff(w))[:count])
    return [(0.5 * (w[i] + w[i + 1]), int(i) + 1) for i in g]


def _forms(f):
    def factorize(detection):
        f.set_null_pivot_detection(detection)

        def run(sigma):
            assert f.factorize(1.0, -sigma)
            return f.inertia()
        return run

    return [factorize(True), lambda s: f.count(1.0, -s, True), lambda s: f.count(1.0, -s, False)]


@pytest.mark.parametrize("precision", [0, 1])
def test_each_form_is_replayed_from_its_eighth_use(precision):
    from hsolve_b200 import Factorization

    f = Factorization(device=0, precision=precision)
    replays = 0
    for nx, ny in ((23, 17), (31, 19)):
        a = laplacian_2d(nx, ny)
        w = np.linalg.eigvalsh(a.toarray())
        shifts = _gaps(w, 13)
        f.analyze(a, None, 1.0, 0.0)
        assert f.graph_stats()["factor_graphs"] == 0  # the work of the analysis before is gone
        uses, graphs = {}, set()
        for form, run in enumerate(_forms(f)):
            for t in range(4 * USES):
                sigma, below = shifts[(5 * t) % len(shifts)]
                c = run(sigma)
                assert (c.neg, c.zero, c.pos) == (below, 0, w.size - below)
                uses[form] = uses.get(form, 0) + 1
                if uses[form] >= USES:
                    replays += 1
                    graphs.add(form)
                if c.replans:  # delayed pivots: the pass was run again, directly, on a new plan
                    uses, graphs = {form: 1}, set()
                s = f.graph_stats()
                assert (s["factor_graphs"], s["factor_replays"]) == (len(graphs), replays)
            assert form in graphs


@pytest.mark.parametrize("n", [LARGEST, LARGEST + 1])
def test_orders_around_the_largest_captured(n):
    from hsolve_b200 import Factorization

    f = Factorization(device=0)
    f.analyze(laplacian_1d(n), None, 1.0, 0.0)
    for _ in range(USES + 1):
        c = f.count(1.0, 0.0)
        assert (c.neg, c.zero, c.pos) == (0, 0, n)
    assert f.graph_stats()["factor_replays"] == (2 if n <= LARGEST else 0)


def test_captured_solves_are_bounded():
    from hsolve_b200 import Factorization

    a = laplacian_2d(9, 7)
    f = Factorization(device=0)
    f.analyze(a, None, 1.0, 0.0)
    assert f.factorize(1.0, 0.0)
    b = np.random.default_rng(2).standard_normal((a.shape[0], 150))
    want = np.linalg.solve(a.toarray(), b)
    for p in [*range(1, 151), 150, 3, 149, 1]:  # each width moves the work arrays up to 150
        x = f.solve(b[:, :p])
        # a symmetric positive definite matrix with a condition below 100
        assert np.abs(x - want[:, :p]).max() <= 100 * a.shape[0] * np.finfo(float).eps * np.abs(want).max()
        assert f.graph_stats()["solve_graphs"] <= SOLVE_GRAPHS
    assert f.graph_stats()["solve_graphs"] == SOLVE_GRAPHS
    assert f.graph_stats()["solve_replays"] == 154


def test_two_threads_replay_their_own_objects():
    from hsolve_b200 import Factorization

    a = laplacian_2d(29, 23)
    n = a.shape[0]
    shifts = _gaps(np.linalg.eigvalsh(a.toarray()), 3 * USES)
    b = np.random.default_rng(5).standard_normal((n, 3))

    def work(mine, out):
        f = Factorization(device=0)
        f.analyze(a, None, 1.0, 0.0)
        for sigma, below in mine:
            assert f.factorize(1.0, -sigma)
            out.append((f.inertia().neg - below, f.solve(b)))
        assert f.graph_stats()["factor_replays"] == len(mine) - USES + 1

    serial, threaded = [[], []], [[], []]
    for t in range(2):
        work(shifts[t::2], serial[t])
    threads = [threading.Thread(target=work, args=(shifts[t::2], threaded[t])) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, t in zip(serial, threaded):
        assert len(s) == len(t) == len(shifts) // 2
        for (ds, xs), (dt, xt) in zip(s, t):
            assert ds == dt == 0
            np.testing.assert_array_equal(xs, xt)  # fixed orders of summation


def test_concurrent_shifts_of_a_session():
    import hsolve_b200
    from hsolve_b200.gen import yee
    from oracle import yee_exact

    box = yee.Box((8, 7, 6))
    a, _ = yee.pencil(box)
    w = yee_exact.exact_spectrum(box.cells)
    lo, hi = (0.5 * (w[i] + w[i - 1]) for i in (np.searchsorted(w, 30.0), np.searchsorted(w, 150.0)))
    inside = w[(w > lo) & (w < hi)]
    session = hsolve_b200.Session(a)
    for _ in range(USES + 4):
        r = session.solve(lower=lo, upper=hi)
        assert r.success and r.report["certificate"]["passed"]
        np.testing.assert_allclose(np.sort(r.eigenvalues), inside, rtol=1e-10)
