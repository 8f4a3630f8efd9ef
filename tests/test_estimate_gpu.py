"""The predicted device memory of a factorization holds what a dense front's pivoting takes beside its panel."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [70, 300, 2047, 2048])
def test_scratch_of_a_dense_front(n, precision):
    from hsolve_b200 import Factorization

    a = sp.csr_matrix(np.ones((n, n)) + n * np.eye(n))
    f = Factorization(device=0, precision=precision)
    f.analyze(a, None, 1.0, 0.0)
    e = f.estimate()
    assert (e["supernodes"], e["factor_entries"]) == (1, n * n)
    # the panel in the factor's type, values and scaling of the pencil, and in doubles the rows of a panel of 32
    # pivots beside those of the pending pivots (up to 128, in fronts of 2,048 rows and more 224), a control block and
    # two sets of two 32 x 32 blocks, labels, types and maxima
    pending = min(n, 224 if n >= 2048 else 128)
    scratch = n * (32 + pending) + 8 + 2 * (2 * 32 * 32 + 16 + 4 + 2 * 32)
    need = (8 >> precision) * n * n + 32 * (n * (n + 1) // 2 + n) + 8 * scratch
    assert need <= 1e6 * e["device_mb"] <= 1.2 * need
