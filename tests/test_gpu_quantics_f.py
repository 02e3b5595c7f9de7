"""Registered quantics functions at lengths around the 53 binary digits that one
integer holds, and tiny factorizations of them, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,fid,params,d", [("qtt1d", "F_QTT1D", [0], 2), ("qtt1d", "F_QTT1D", [2], 2),
                                               ("qtt2d", "F_QTT2D", [], 4)])
@pytest.mark.parametrize("L", [2, 31, 32, 33, 52, 53, 54, 70])
def test_values(T, oracle, name, fid, params, d, L):
    rng = np.random.default_rng(L)
    pts = rng.integers(1, d + 1, size=(300, L))
    pts[0], pts[1] = 1, d
    got = T.feval(T.DeviceFunction(name, params), [d] * L, pts)
    assert np.array_equal(got, oracle.feval(getattr(oracle, fid), params, pts))


@pytest.mark.parametrize("L,maxbond", [(3, 2), (5, 1), (9, 7), (40, 6)])
def test_small_solves(T, oracle, L, maxbond):
    kw = dict(tolerance=1e-12, maxbonddim=maxbond, maxiter=4)
    tci, ranks, errors = T.crossinterpolate2(float, T.DeviceFunction("qtt1d", [0]), [2] * L, **kw)
    ref, rranks, rerrors = oracle.crossinterpolate2([2] * L, oracle.F_QTT1D, [0], **kw)
    assert list(ranks) == list(rranks) and np.array_equal(errors, rerrors)
    for b in range(1, L + 1):
        assert np.array_equal(tci.sitetensor(b), ref.core(b))
