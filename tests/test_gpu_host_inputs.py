"""Large host inputs taken in place by the device: batches of matrices in every
memory order, and points packed and range-checked on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batched_matrices_of_any_order(T, oracle):
    rng = np.random.default_rng(2)
    mats = []
    for k in range(60):
        a = rng.standard_normal((5 + 2 * k, 4 + 3 * (k % 17)))
        mats.append([a, np.asfortranarray(a), np.asfortranarray(a)[::2, 1:], a.T, a.astype(np.float32)][k % 5])
    got = T.rrlu_batched(mats, maxrank=20)
    for a, (rows, cols, K, err) in zip(mats, got):
        r = oracle.rrlu(np.asarray(a, np.float64), maxrank=20)
        assert K == r["npivot"] and err == r["error"]
        assert np.array_equal(rows - 1, r["rowpermutation"][:K]) and np.array_equal(cols - 1, r["colpermutation"][:K])


@pytest.mark.parametrize("precision", ["fp64", "tf32x3"])
@pytest.mark.parametrize("n", [10, 6553, 6554, 20000])  # ten sites: the device packs from 65536 values on
def test_points(T, precision, n):
    rng = np.random.default_rng(n)
    dims = [2, 3, 4, 5, 2, 3, 4, 5, 2, 3]
    bonds = [1, 2, 5, 7, 8, 9, 8, 7, 5, 2, 1]
    tt = T.TensorTrain([rng.standard_normal((bonds[s], dims[s], bonds[s + 1])) for s in range(10)])
    pts = np.stack([rng.integers(1, d + 1, size=n) for d in dims], axis=1)
    got = tt.evaluate(pts, precision=precision)
    one = np.array([tt.evaluate(pts[k:k + 1], precision=precision)[0] for k in range(0, n, max(1, n // 7))])
    assert np.array_equal(got[::max(1, n // 7)], one)
    for k, site, v in ((0, 0, 3), (n - 1, 9, 4), (n // 2, 3, 0), (n // 3, 5, -7), (n // 3, 2, 1 << 40)):
        bad = pts.copy()
        bad[k, site] = v
        with pytest.raises(T.ArgumentError, match="out of range"):
            tt.evaluate(bad, precision=precision)
