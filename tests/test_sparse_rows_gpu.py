"""hsg_spmm and hsg_shifted_residual around the row lengths at which their kernels change (four lanes a
row up to 128 entries, the warp beyond), ragged numbers of rows and every column width, against numpy."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _rows(n, lengths, rng):
    """A matrix whose row i has min(lengths[i % len], n) entries."""
    rows, cols = [], []
    for i in range(n):
        k = min(lengths[i % len(lengths)], n)
        c = rng.choice(n, size=k, replace=False)
        rows += [i] * k
        cols += list(c)
    return sp.csr_matrix((rng.standard_normal(len(rows)), (rows, cols)), shape=(n, n))


def _dev(x):
    import torch

    return torch.from_numpy(np.ascontiguousarray(x.T)).cuda()


LENGTHS = [[0, 1, 3, 4, 5, 13], [127, 128, 129, 2, 0, 7, 300], [1], [600, 1, 1, 1, 1, 1, 1, 1, 1]]


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 700])
@pytest.mark.parametrize("lengths", range(len(LENGTHS)))
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5, 8, 9, 16])
def test_rows(n, lengths, p):
    import torch

    from hsolve_b200 import _native

    # the reference in extended precision: a double reference rounds x + sigma y by itself
    big = lambda m: m.toarray().astype(np.longdouble)  # noqa: E731
    rng = np.random.default_rng(n + 31 * lengths + p)
    a, b = _rows(n, LENGTHS[lengths], rng), _rows(n, LENGTHS[lengths][::-1], rng)
    if not a.nnz or not b.nnz:
        pytest.skip("a matrix without entries has no arrays to point to: the calls refuse it")
    x, y, z = (rng.standard_normal((n, p)) for _ in range(3))
    sigma = 0.7
    da, db = _native.DeviceCsr(a), _native.DeviceCsr(b)
    long = 2 + max(a.getnnz(axis=1).max(), b.getnnz(axis=1).max())
    # Y = 2 A X - 0.5 Z: a sum of `long` products, each rounded
    out = _dev(z)
    _native.spmm_device(da, _dev(x), out, 2.0, -0.5)
    size = 2 * (abs(a) @ abs(x)) + 0.5 * abs(z)
    want = 2 * (big(a) @ x) - 0.5 * z
    assert (np.abs(out.cpu().numpy().T - want) <= 2 * long * EPS * size).all()
    for bb, dbb in ((b, db), (sp.identity(n, format="csr"), None)):
        w = x + np.longdouble(sigma) * y
        r, s = big(bb) @ w - big(a) @ y, abs(big(bb)) @ abs(w) + abs(big(a)) @ abs(y)
        got, om = torch.empty(p, n, dtype=torch.float64, device="cuda"), torch.empty(p, dtype=torch.float64, device="cuda")
        _native.shifted_residual_device(da, dbb, sigma, _dev(x), _dev(y), got, om)
        assert (np.abs(got.cpu().numpy().T - r) <= 2 * long * EPS * s).all()
        want = np.max(np.where(s > 0, np.abs(r) / np.where(s > 0, s, 1.0), 0.0), axis=0)
        np.testing.assert_allclose(om.cpu().numpy(), want.astype(float), rtol=0, atol=4 * long * EPS)


def test_backward_error_of_rows_that_are_not_finite():
    import torch

    from hsolve_b200 import _native

    a = sp.identity(9, format="csr")
    for value in (np.inf, np.nan):
        x, y = np.ones((9, 3)), np.ones((9, 3))
        y[4, 1] = value
        om = torch.empty(3, dtype=torch.float64, device="cuda")
        _native.shifted_residual_device(_native.DeviceCsr(a), None, 0.5, _dev(x), _dev(y), None, om)
        assert np.isinf(om.cpu().numpy()[1]) and np.isfinite(om.cpu().numpy()[[0, 2]]).all()
