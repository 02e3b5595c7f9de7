"""rrlu_batched of matrices taken where they are, copied into one array, or copied one
after the other, by their mean size: every memory order, type and alignment in one batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _variants(a):
    buf = np.zeros(a.nbytes + 16, np.uint8)
    off = buf[4:4 + a.nbytes].view(np.float64).reshape(a.shape, order="F")
    off[...] = a
    wide = np.zeros((a.shape[0] * 2, a.shape[1] + 1))
    wide[::2, 1:] = a
    return [np.asfortranarray(a), np.ascontiguousarray(a), off, wide[::2, 1:], np.asfortranarray(a)[:, ::-1],
            a.astype(np.float32), np.ascontiguousarray(a.T).T]


@pytest.mark.parametrize("mean", ["small", "at the line", "large"])
def test_bits(T, oracle, mean):
    rng = np.random.default_rng(4)
    m, n = {"small": (11, 17), "at the line": (32, 64), "large": (60, 70)}[mean]
    mats = []
    for k in range(3):
        mats += _variants(rng.standard_normal((m + k, n)))
    if mean == "large":
        mats += [np.zeros((0, 5)), np.zeros((4, 0)), np.ones((1, 1))]
    got = T.rrlu_batched(mats, maxrank=9)
    for a, (rows, cols, K, err) in zip(mats, got):
        if a.size == 0:
            assert K == 0 and len(rows) == 0
            continue
        r = oracle.rrlu(np.asarray(a, np.float64), maxrank=9)
        assert K == r["npivot"] and err == r["error"]
        assert np.array_equal(rows - 1, r["rowpermutation"][:K]) and np.array_equal(cols - 1, r["colpermutation"][:K])
    for row_major in (False, True):  # one order only
        same = [np.array(a, np.float64, order="C" if row_major else "F") for a in mats[:7]]
        for x, y in zip(T.rrlu_batched(same, maxrank=9), got):
            assert x[2:] == y[2:] and np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])
