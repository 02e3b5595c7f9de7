"""rrlu of matrices with NaN, infinities and zeros on each of its kernels (one warp, one
CTA, a cluster, every SM): the NaN error exactly where the oracle has it, and no other
error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left", [True, False])
@pytest.mark.parametrize("kind", ["normal", "zeros", "inf", "one nan", "nan row", "nan column", "all nan"])
@pytest.mark.parametrize("shape", [(7, 9), (30, 30), (60, 70), (530, 517)])
def test_nan(T, oracle, shape, kind, left):
    rng = np.random.default_rng(shape[0])
    A = rng.standard_normal(shape)
    if kind == "zeros":
        A[rng.random(shape) < 0.9] = 0.0
    elif kind == "inf":
        A[3, 4] = np.inf
    elif kind == "one nan":
        A[4, 3] = np.nan
    elif kind == "nan row":
        A[5, :] = np.nan
    elif kind == "nan column":
        A[:, 2] = np.nan
    elif kind == "all nan":
        A[...] = np.nan
    for maxrank in (2, 12):
        kw = dict(maxrank=maxrank, leftorthogonal=left)
        want = None
        try:
            want = oracle.rrlu(A, **kw)
        except oracle.OracleError as e:
            assert kind not in ("normal", "zeros") and "NaN" in str(e)
        if want is None:
            with pytest.raises(T.TCIError, match="NaN") as err:
                T.rrlu(A, **kw)
            assert err.value.code == T.TCI_ERR_NAN
            continue
        g = T.rrlu(A, **kw)
        assert g.npivot == want["npivot"] and np.array_equal(g.error, want["error"], equal_nan=True)
        assert np.array_equal(g.rowpermutation - 1, want["rowpermutation"])
        assert np.array_equal(g.colpermutation - 1, want["colpermutation"])
        assert np.array_equal(g.L, want["L"], equal_nan=True) and np.array_equal(g.U, want["U"], equal_nan=True)
    if kind in ("all nan", "nan row", "nan column"):
        with pytest.raises(oracle.OracleError):
            oracle.rrlu(A, leftorthogonal=left)
        with pytest.raises(T.TCIError, match="NaN"):
            T.rrlu(A, leftorthogonal=left)
