"""FP64 evaluation of trains (tt_eval.cu): bits against the same sums in the
same order on the host, at the edges of its point blocks and output groups and
for core values of every class (dense, zeros and ones, outside the integer
range)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(cores, pts):
    v = np.ones((pts.shape[0], 1))
    for s, c in enumerate(cores):
        m = c[:, pts[:, s] - 1, :]  # r0 x np x r1
        acc = np.zeros((pts.shape[0], c.shape[2]))
        with np.errstate(over="ignore", invalid="ignore"):
            for t in range(c.shape[0]):
                acc = acc + v[:, t:t + 1] * m[t]
        v = acc
    return v[:, 0]


def _cores(bonds, d, kind, rng):
    out = []
    for s in range(len(bonds) - 1):
        c = rng.standard_normal((bonds[s], d, bonds[s + 1]))
        if kind == "unit" and s % 2:  # rows of a unit matrix, as in a cross-interpolated train
            c[:, 0, :] = np.eye(bonds[s], bonds[s + 1])
            c[:, 1, :] *= rng.random(c[:, 1, :].shape) < 0.5
        if kind == "extreme" and s == 1:
            c *= 10.0 ** rng.integers(-250, 60, size=c.shape)
        out.append(c)
    return out


@pytest.mark.parametrize("kind", ["dense", "unit", "extreme"])
@pytest.mark.parametrize("bonds", [(1, 1), (1, 2, 1), (1, 3, 4, 1), (1, 5, 17, 6, 1), (1, 16, 33, 16, 1),
                                   (1, 7, 130, 80, 9, 1)])
def test_bits(T, bonds, kind):
    rng = np.random.default_rng(len(bonds) * 31 + bonds[1])
    d = 4
    cores = _cores(bonds, d, kind, rng)
    for n in (1, 3, 260, 2500):
        pts = rng.integers(1, d + 1, size=(n, len(cores)))
        got, want = T.TensorTrain(cores).evaluate(pts), _reference(cores, pts)
        assert np.array_equal(got, want, equal_nan=True), (n, np.abs(got - want).max())
