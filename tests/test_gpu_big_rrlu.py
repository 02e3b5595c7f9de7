"""Factorizations spread over every SM: pivots that need the comparison of squares
(values near the ends of the range, near ties), NaN and all-NaN rows, ragged blocks,
against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(530, 517), (2049, 130), (131, 2100), (65, 4097)])
@pytest.mark.parametrize("kind", ["normal", "tiny", "huge", "ties", "nan", "zeros"])
def test_pivots(T, oracle, shape, kind):
    rng = np.random.default_rng(shape[0])
    A = rng.standard_normal(shape)
    if kind == "tiny":
        A *= 1e-160
    elif kind == "huge":
        A *= 1e155
    elif kind == "ties":
        A = (1.0 + rng.integers(-12, 13, size=shape) * 2.0 ** -52) * rng.choice([-1.0, 1.0], size=shape)
    elif kind == "nan":
        A[7, :] = np.nan
    elif kind == "zeros":
        A[rng.random(shape) < 0.9] = 0.0
    for left in (True, False):
        kw = dict(maxrank=14, leftorthogonal=left)
        try:
            r = oracle.rrlu(A, **kw)
        except Exception:
            with pytest.raises(Exception):
                T.rrlu(A, **kw)
            continue
        g = T.rrlu(A, **kw)
        assert g.npivot == r["npivot"] and np.array_equal(g.error, r["error"], equal_nan=True)
        assert np.array_equal(g.rowpermutation - 1, r["rowpermutation"])
        assert np.array_equal(g.colpermutation - 1, r["colpermutation"])
        assert np.array_equal(g.L, r["L"], equal_nan=True) and np.array_equal(g.U, r["U"], equal_nan=True)
