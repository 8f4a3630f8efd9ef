"""A captured solve or factorization counts its own launches at each replay, also where another thread launched
kernels while it was captured."""
import threading

import numpy as np
import pytest

from helpers import laplacian_2d

pytestmark = pytest.mark.gpu


def _replay_counts(a, widths):
    """Kernel launches of one replayed solve of each width, of a new object (each width is captured here)."""
    from hsolve_b200 import Factorization, _native

    n = a.shape[0]
    f = Factorization(device=0)
    f.analyze(a, None, 1.0, 0.0)
    assert f.factorize(1.0, -0.1)

    def counts():
        out = []
        for p in widths:
            b = np.ones((n, p))
            before = _native.kernel_launches()
            f.solve(b)
            out.append(_native.kernel_launches() - before)
        return out

    f.solve(np.ones((n, max(widths))))  # the work arrays of the widest solve, and the solve operators
    counts()
    return counts


def test_replays_count_their_own_launches():
    import torch

    from hsolve_b200 import _native

    a = laplacian_2d(23, 17)
    widths = range(1, 9)
    alone = _replay_counts(a, widths)()
    assert min(alone) > 0
    m, x = _native.DeviceCsr(a), torch.ones(1, a.shape[0], dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    stop, started = threading.Event(), threading.Event()

    def launch():
        while not stop.is_set():
            _native.spmm_device(m, x, y)
            started.set()

    t = threading.Thread(target=launch)
    t.start()
    assert started.wait(30)
    try:
        counts = _replay_counts(a, widths)
    finally:
        stop.set()
        t.join()
    assert counts() == alone
