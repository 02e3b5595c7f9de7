"""The FP64 contraction kernel (contract.cu) through matmul: bits against the
same sums in the same order, at the edges of its tiles and slices and for values
of every class (dense, exact zeros and ones, outside the integer range)."""
import numpy as np
import pytest

from test_gpu_int_products import _matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["normal", "zeros", "extreme", "integers"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (64, 64, 16), (65, 63, 17), (128, 32, 15), (129, 33, 33), (257, 16, 48),
                                   (255, 15, 5), (5, 300, 70), (300, 3, 100), (400, 390, 31)])
def test_bits(T, shape, kind):
    M, N, K = shape
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    A, B = _matrix(kind, M, K, rng), _matrix(kind, K, N, rng)
    if kind == "zeros":  # whole slices stay dense beside slices with zeros
        A[:, 16:32] = rng.standard_normal((M, max(0, min(K, 32) - 16)))
        B[16:32] = rng.standard_normal((max(0, min(K, 32) - 16), N))
    want = np.zeros((M, N))
    with np.errstate(over="ignore", invalid="ignore"):
        for k in range(K):
            want = want + A[:, k:k + 1] * B[k]
    C, _ = T.matmul(A, B)
    assert np.array_equal(C, want, equal_nan=True)
