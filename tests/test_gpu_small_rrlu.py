"""Factorizations finished by one warp: shapes around its 32 scaled lines and the
eight rows of its smaller tiles, both directions, with ties, zeros and NaN, against
the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 5), (5, 1), (2, 2), (7, 9), (8, 8), (9, 8), (13, 14), (16, 12), (17, 11), (24, 24),
                                   (31, 6), (32, 6), (33, 5), (6, 31), (6, 32), (5, 33), (96, 2), (2, 96), (40, 40)])
@pytest.mark.parametrize("kind", ["normal", "integers", "zeros", "nan"])
def test_shapes(T, oracle, shape, kind):
    rng = np.random.default_rng(shape[0] * 100 + shape[1])
    A = rng.standard_normal(shape)
    if kind == "integers":
        A = rng.integers(-2, 3, size=shape).astype(np.float64)
    elif kind == "zeros":
        A[rng.random(shape) < 0.6] = 0.0
    elif kind == "nan":
        A[shape[0] // 2, shape[1] // 2] = np.nan
    for left in (True, False):
        kw = dict(leftorthogonal=left, reltol=1e-14)
        try:
            r = oracle.rrlu(A, **kw)
        except Exception as e:
            with pytest.raises(Exception):
                T.rrlu(A, **kw)
            continue
        g = T.rrlu(A, **kw)
        assert g.npivot == r["npivot"] and np.array_equal(g.error, r["error"], equal_nan=True)
        assert np.array_equal(g.rowpermutation - 1, r["rowpermutation"])
        assert np.array_equal(g.colpermutation - 1, r["colpermutation"])
        assert np.array_equal(g.L, r["L"], equal_nan=True) and np.array_equal(g.U, r["U"], equal_nan=True)
