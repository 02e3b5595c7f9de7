"""The copies of rrlu's L and U: equal to numpy's in values, order and ownership, at the
edges of the column blocks and of the threaded range."""
import threading

import numpy as np
import pytest

from tci_gb300 import _own_copy


@pytest.mark.parametrize("shape", [(0, 0), (0, 5), (5, 0), (1, 1), (1, 8192), (1, 8193), (3, 5000), (16, 512), (16, 513),
                                   (511, 40), (512, 16), (512, 17), (512, 1000), (513, 40), (900, 444), (900, 445)])
def test_copy(shape):
    a = np.arange(shape[0] * shape[1], dtype=np.float64).reshape(shape, order="F")
    b = _own_copy(a)
    assert np.array_equal(a, b) and b.flags.c_contiguous and b.flags.owndata and b.dtype == a.dtype
    assert not np.shares_memory(a, b)


@pytest.mark.parametrize("allowed", [0, 1, 2, 3])
def test_copy_without_threads(monkeypatch, allowed):
    """As many threads as the system gives."""
    left = [allowed]
    start = threading.Thread.start

    def limited(self):
        if not left[0]:
            raise RuntimeError("can't start new thread")
        left[0] -= 1
        start(self)

    monkeypatch.setattr(threading.Thread, "start", limited)
    a = np.random.default_rng(1).standard_normal((700, 601)).T.copy().T
    assert np.array_equal(_own_copy(a), a)
