"""The registered "served" function with centres so far away that their squares leave
the 64-bit integers: f, solves and searches use double sums there.  Reference in plain
numpy; the library's exponential and numpy's agree to a few units in the last place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _f(prm, pts):
    a0, a1 = np.zeros(len(pts)), np.zeros(len(pts))
    for s in range(pts.shape[1]):
        a0 = a0 + pts[:, s].astype(float) ** 2
        a1 = a1 + (pts[:, s] - np.trunc(prm[3 + s])) ** 2
    return 1.0 / (1.0 + prm[0] * a0) + prm[1] * np.exp(-prm[2] * a1)


@pytest.mark.parametrize("c,g", [(3.0, 0.1), (2.9, 0.1), (-1.5, 0.05), (600.0, 1e-6), (3e9, 1e-20), (4e9, 1e-20),
                                 (-5e9, 1e-20), (1e30, 1e-62)])
def test_values_solve_and_search(T, c, g):
    dims = [6, 5, 4, 6]
    prm = [0.3, 2.0, g] + [c + 0.0 * s if abs(c) > 1e6 else c + s for s in range(4)]
    if abs(c) >= 2.0 ** 62:
        prm[3:] = [2.0 ** 62] * 4  # the conversion to 64 bits ends there
        prm[2] = 1e-38
    f = T.DeviceFunction("served", prm)
    pts = np.stack(np.meshgrid(*[np.arange(1, d + 1) for d in dims], indexing="ij"), -1).reshape(-1, 4)
    want = _f(prm, pts)
    assert np.abs(T.feval(f, dims, pts) - want).max() <= 1e-14 * np.abs(want).max()
    tci, _, _ = T.crossinterpolate2(float, f, dims, tolerance=1e-10)
    got = tci.evaluate(pts)
    assert np.abs(got - want).max() <= 1e-8 * np.abs(want).max()
    at = {tuple(p): k for k, p in enumerate(pts)}
    for p, e in tci.estimatetrueerror(nsearch=8, seed=1):
        k = at[tuple(p)]
        assert abs(e - abs(want[k] - got[k])) <= 1e-13 * np.abs(want).max()
    pivot = T.optfirstpivot(f, dims)
    assert want[at[tuple(int(x) for x in pivot)]] >= want[0]
