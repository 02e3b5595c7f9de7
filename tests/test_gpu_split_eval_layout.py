"""Split-precision train evaluation where its shared and tensor memory change size.

A point's value comes from the same products in the same order whatever else is
evaluated with it, so subsets agree bit for bit; against FP64 the bound is that of
split products accumulated in FP32: 1e-5 per site, relative to the largest value.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,bonds,points", [
    (2, [1, 1, 1], 129),  # one column block of 32
    (2, [2, 12, 16, 3], 100001),  # five CTAs per SM, more than one tile each
    (3, [3, 17, 33, 8, 2], 127),  # 96 columns; odd bonds around the 8- and 32-deep edges
    (2, [2, 31, 32, 33, 64, 7], 70001),  # 128 columns, two chunks
    (4, [4, 65, 9, 96, 5], 1),  # 384 columns: one CTA per SM
    (32, [16, 16], 20001),  # 512 columns with the smallest chunks
    (4, [4, 127, 128, 128, 4], 40001),  # everything at its largest
])
def test_split_evaluate_layouts(T, oracle, d, bonds, points):
    rng = np.random.default_rng(d + sum(bonds))
    b = [1] + bonds + [1]
    cores = [rng.standard_normal((b[n], d, b[n + 1])) / np.sqrt(b[n] * d) for n in range(len(b) - 1)]
    L = len(cores)
    pts = rng.integers(1, d + 1, size=(points, L))
    tt = T.TensorTrain(cores)
    got = tt.evaluate(pts, precision="tf32x3")
    ref = tt.evaluate(pts)
    some = rng.permutation(points)[:200]
    np.testing.assert_allclose(ref[some], oracle.tt_evaluate(cores, pts[some]), rtol=1e-11, atol=1e-13)
    assert np.abs(got - ref).max() <= 1e-5 * L * np.abs(ref).max()
    assert np.array_equal(tt.evaluate(pts[some], precision="tf32x3"), got[some])
