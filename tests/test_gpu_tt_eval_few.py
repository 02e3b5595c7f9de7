"""FP64 train evaluation at few points, where a thread takes one output: bits against
the same sums in the same order, at the edges of its blocks of eight terms and of the
rules for that form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(kind, shape, rng):
    a = rng.standard_normal(shape)
    if kind == "zeros":
        a[rng.random(shape) < 0.4] = 0.0
        a[rng.random(shape) < 0.2] = 1.0
    elif kind == "extreme":
        a *= 10.0 ** rng.integers(-160, 120, size=shape)
        a.flat[0] = np.inf
    return a


@pytest.mark.parametrize("kind", ["normal", "zeros", "extreme"])
@pytest.mark.parametrize("r", [1, 7, 8, 9, 31, 33, 127, 128, 129, 511, 512, 513])
@pytest.mark.parametrize("n", [1, 3, 400])
def test_bits(T, kind, r, n):
    rng = np.random.default_rng(r + n)
    d = 3
    cores = [_values(kind, s, rng) for s in ((1, d, r), (r, d, max(1, r - 1)), (max(1, r - 1), d, 5), (5, d, 1))]
    pts = rng.integers(1, d + 1, size=(n, 4))
    want = np.ones((n, 1))
    with np.errstate(all="ignore"):
        for s, c in enumerate(cores):
            sl = c[:, pts[:, s] - 1, :]  # (r0, points, r1)
            w = np.zeros((n, c.shape[2]))
            for t in range(c.shape[0]):
                w = w + want[:, t:t + 1] * sl[t]
            want = w
    got = T.TensorTrain(cores).evaluate(pts)
    assert np.array_equal(got, want[:, 0], equal_nan=True)
