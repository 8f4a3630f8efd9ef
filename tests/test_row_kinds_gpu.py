"""hsg_spmm and hsg_shifted_residual around the entries a row at which their kernels take four lanes a row, sixteen
or a warp, in chunks of 16 and 64 rows, with rows of different kinds beside each other, against numpy; and that
neighbouring long rows are as quick as spread ones."""
import time

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
SMALL = 444 * 16  # most rows that are taken in chunks of 16


def _matrix(counts, n, rng):
    """Row i has counts[i] entries, in consecutive columns around the diagonal (cyclically)."""
    counts = np.minimum(counts, n)
    rows = np.repeat(np.arange(n), counts)
    start = np.arange(n) - counts // 2
    cols = (np.repeat(start, counts) + np.arange(counts.sum()) - np.repeat(np.cumsum(counts) - counts, counts)) % n
    return sp.csr_matrix((rng.standard_normal(counts.sum()), (rows, cols)), shape=(n, n))


def _dev(x):
    import torch

    return torch.from_numpy(np.ascontiguousarray(x.T)).cuda()


def _check(a, b, p, rng):
    import torch

    from hsolve_b200 import _native

    n = a.shape[0]
    x, y, z = (rng.standard_normal((n, p)) for _ in range(3))
    sigma = 0.7
    da, db = _native.DeviceCsr(a), _native.DeviceCsr(b)
    # every sum: at most `long` products, each rounded, on either side
    long = 4 + a.getnnz(axis=1).max() + b.getnnz(axis=1).max()
    out = _dev(z)
    _native.spmm_device(da, _dev(x), out, 2.0, -0.5)
    size = 2 * (abs(a) @ abs(x)) + 0.5 * abs(z)
    assert (np.abs(out.cpu().numpy().T - (2 * (a @ x) - 0.5 * z)) <= 4 * long * EPS * size).all()
    for bb, dbb in ((b, db), (sp.identity(n, format="csr"), None)):
        w = x + sigma * y
        r, s = bb @ w - a @ y, abs(bb) @ abs(w) + abs(a) @ abs(y)
        got = torch.full((p, n), np.nan, dtype=torch.float64, device="cuda")
        om = torch.full((p,), np.nan, dtype=torch.float64, device="cuda")
        _native.shifted_residual_device(da, dbb, sigma, _dev(x), _dev(y), got, om)
        got = got.cpu().numpy().T
        assert (np.abs(got - r) <= 4 * long * EPS * s).all()
        want = np.max(np.where(s > 0, np.abs(got) / np.where(s > 0, s, 1.0), 0.0), axis=0)
        np.testing.assert_allclose(om.cpu().numpy(), want, rtol=4 * long * EPS, atol=0)


@pytest.mark.parametrize("p", [1, 2, 3, 8, 9])
@pytest.mark.parametrize("entries", [24, 25, 96, 97, 128, 129, 512, 513])
@pytest.mark.parametrize("n", [1030, SMALL + 33])
def test_entries_a_row(n, entries, p):
    rng = np.random.default_rng(n + entries + p)
    _check(_matrix(np.full(n, entries), n, rng), _matrix(np.full(n, 3), n, rng), p, rng)


@pytest.mark.parametrize("p", [1, 2, 3, 8, 9])
@pytest.mark.parametrize("n", [15, 16, 17, 640, SMALL, SMALL + 1, SMALL + 63])
def test_rows_of_all_kinds(n, p):
    """Chunks of short rows, of wide ones, a block of neighbouring long rows, long rows alone and empty rows; the
    second matrix has its long rows elsewhere."""
    rng = np.random.default_rng(n + p)
    counts = np.full(n, 5)
    counts[n // 3:n // 3 + 130] = 140
    counts[n // 2:n // 2 + 21] = 700
    counts[-1] = 3 * n
    counts[1::50] = 0
    other = np.full(n, 1)
    other[:9] = 600
    _check(_matrix(counts, n, rng), _matrix(other, n, rng), p, rng)


def test_many_chunks():
    """Long rows at both ends of 4,738 chunks of 64."""
    n = 4736 * 64 + 77
    rng = np.random.default_rng(1)
    counts = np.full(n, 3)
    counts[-5:] = 2000
    counts[7] = 900
    _check(_matrix(counts, n, rng), _matrix(np.full(n, 1), n, rng), 2, rng)


@pytest.mark.parametrize("p", [1, 8])
def test_neighbouring_long_rows_are_shared(p):
    """Eight full rows of 3,000 beside each other take at most twice the time of eight that lie apart (five times
    where one warp takes them one after another)."""
    import torch

    from hsolve_b200 import _native

    n, rng = 3000, np.random.default_rng(2)
    x = torch.ones(p, n, dtype=torch.float64, device="cuda")
    r, om = torch.empty_like(x), torch.empty(p, dtype=torch.float64, device="cuda")

    def best(rows):
        counts = np.full(n, 13)
        counts[rows] = n
        m = _native.DeviceCsr(_matrix(counts, n, rng))
        times = []
        for _ in range(30):
            t = time.perf_counter()
            _native.spmm_device(m, x, r)
            _native.shifted_residual_device(m, m, 0.7, x, x, r, om)
            times.append(time.perf_counter() - t)
        return min(times)

    assert best(np.arange(n - 8, n)) <= 2.0 * best(np.arange(8) * (n // 8) + 100)
