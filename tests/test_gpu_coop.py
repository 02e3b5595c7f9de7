"""Single solves whose bond factorizations run on a thread-block cluster beside
the resident kernel, and rrlu of host matrices on a cluster: bits against the
oracle around the sizes where the route changes, for each registered f."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,fid,params,dims,tol,mbd", [
    ("lorentz", "F_LORENTZ", [1.5], [10] * 6, 1e-10, 200),      # tables, bonds up to 120 x 120
    ("lorentz", "F_LORENTZ", [1.0], [3, 7, 2, 11, 5, 4], 1e-9, 7),  # uneven sites, capped rank
    ("served", "F_SERVED", [0.3, 0.7, 0.2, 3, 1, 4, 1, 5], [8] * 5, 1e-9, 64),
    ("qtt1d", "F_QTT1D", [0], [2] * 24, 1e-10, 64),             # f evaluated directly
    ("qtt2d", "F_QTT2D", [], [4] * 14, 1e-7, 48),
])
def test_solves(T, oracle, name, fid, params, dims, tol, mbd):
    kw = dict(tolerance=tol, maxbonddim=mbd, maxiter=6)
    g, ranks, errors = T.crossinterpolate2(float, T.DeviceFunction(name, params), dims, **kw)
    r, rranks, rerrors = oracle.crossinterpolate2(dims, getattr(oracle, fid), params, None, **kw)
    assert list(ranks) == list(rranks) and np.array_equal(errors, rerrors)
    assert g.maxsamplevalue == r.maxsamplevalue
    for b in range(1, len(dims) + 1):
        for x, y in zip(g.sets(b), r.sets(b)):
            assert np.array_equal(x, y)
        assert np.array_equal(g.sitetensor(b), r.core(b))


@pytest.mark.parametrize("shape", [(49, 51), (50, 50), (99, 101), (100, 100), (511, 512), (512, 512), (3, 2000),
                                   (20000, 4)])
def test_host_matrices(T, oracle, shape):
    A = np.random.default_rng(shape[0]).standard_normal(shape)
    for left in (True, False):
        g, r = T.rrlu(A, maxrank=60, leftorthogonal=left), oracle.rrlu(A, maxrank=60, leftorthogonal=left)
        assert g.npivot == r["npivot"] and g.error == r["error"]
        assert np.array_equal(g.rowpermutation - 1, r["rowpermutation"])
        assert np.array_equal(g.colpermutation - 1, r["colpermutation"])
        assert np.array_equal(g.L, r["L"]) and np.array_equal(g.U, r["U"])


def test_nan_and_zero(T, oracle):
    A = np.random.default_rng(1).standard_normal((80, 90))
    A[3, 4] = np.inf
    for M in (A, np.zeros((60, 70)), np.full((60, 70), np.nan)):
        try:
            r = oracle.rrlu(M)
        except oracle.OracleError:
            with pytest.raises(T.TCIError, match="NaN"):
                T.rrlu(M)
            continue
        g = T.rrlu(M)
        assert g.npivot == r["npivot"] and np.array_equal(g.rowpermutation - 1, r["rowpermutation"])
        assert np.array_equal(g.L, r["L"], equal_nan=True) and np.array_equal(g.U, r["U"], equal_nan=True)


@pytest.mark.parametrize("L,d,maxbond", [(5, 4, 4), (5, 16, 16), (6, 10, 40), (4, 25, 60)])
def test_caller_f(T, oracle, L, d, maxbond):
    """A caller's f: its factorizations, launched one at a time, against the same
    solve with the values from the registered function."""
    f = T.BatchFunction(lambda p: 1.5 / ((p.astype(np.float64) ** 2).sum(1) + 1.0))
    kw = dict(tolerance=1e-10, maxbonddim=maxbond, maxiter=6)
    got, ranks, errors = T.crossinterpolate2(float, f, [d] * L, **kw)
    ref, rranks, rerrors = oracle.crossinterpolate2([d] * L, oracle.F_LORENTZ, [1.5], **kw)
    assert list(ranks) == list(rranks) and np.array_equal(errors, rerrors)
    for b in range(1, L + 1):
        assert np.array_equal(got.sitetensor(b), ref.core(b))
