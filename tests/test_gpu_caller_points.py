"""Points a caller's f is asked for when a Pi matrix is completed on the device:
sizes around the blocks of the ordering kernels, partly known matrices, and ones
whose points outgrow the buffer handed to f.  Values and pivots against the
oracle bit for bit; no point is asked for twice; order within a call as the
matrix's columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,maxbond,maxiter", [
    ([2, 2], 2, 2),
    ([45, 45], 8, 3),          # 2025 elements
    ([64, 32], 8, 3),          # 2048
    ([241, 17], 3, 2),         # 4097
    ([7, 3, 11, 5], 9, 4),
    ([40, 30, 20], 12, 4),
    ([3] * 12, 20, 4),         # later matrices mostly known
    ([100, 90, 80], 6, 3),     # 8100 x 80 and so on
    ([3, 250, 250, 3], 3, 3),  # up to 562 500 points, more than the buffer unless many are known
    ([2, 256, 256, 4, 2, 2, 2, 2], 2, 3),  # the number of points is needed first
])
def test_points(T, oracle, dims, maxbond, maxiter):
    L, asked = len(dims), []

    def f(p):
        asked.append(np.array(p))
        return 1.5 / ((p.astype(np.float64) ** 2).sum(1) + 1.0)

    kw = dict(tolerance=1e-12, maxbonddim=maxbond, maxiter=maxiter)
    got, ranks, errors = T.crossinterpolate2(float, T.BatchFunction(f), dims, **kw)
    ref, rranks, rerrors = oracle.crossinterpolate2(dims, oracle.F_LORENTZ, [1.5], **kw)
    assert list(ranks) == list(rranks) and np.array_equal(errors, rerrors)
    for b in range(1, L + 1):
        assert np.array_equal(got.sitetensor(b), ref.core(b))
    pts = np.concatenate(asked)
    assert pts.min() >= 1 and (pts <= np.array(dims)).all()
    assert len(np.unique(pts, axis=0)) == len(pts)


def test_order_and_failure(T):
    """The first matrix, all of it unknown, is asked for column by column; an
    exception in f reaches the caller and the next solve is unharmed."""
    asked = []

    def f(p):
        asked.append(np.array(p))
        return 1.0 / (p.sum(1) + 0.5)

    T.crossinterpolate2(float, T.BatchFunction(f), [30, 20], tolerance=1e-9, maxbonddim=4, maxiter=2)
    big = max(asked, key=len)
    assert (np.diff(big[:, 1]) >= 0).all() and (np.diff(big[:, 0])[np.diff(big[:, 1]) == 0] > 0).all()

    def g(p):
        if len(p) > 100:
            raise ValueError("no")
        return 1.0 / (p.sum(1) + 0.5)

    with pytest.raises(ValueError):
        T.crossinterpolate2(float, T.BatchFunction(g), [30, 20], tolerance=1e-9, maxbonddim=4, maxiter=2)
    asked.clear()
    T.crossinterpolate2(float, T.BatchFunction(f), [30, 20], tolerance=1e-9, maxbonddim=4, maxiter=2)
    assert sum(map(len, asked)) == 600
