"""FP64 products on both sides of the line between one thread per output and tiles,
for each tile width, with ragged edges and values of every class, bit for bit."""
import numpy as np
import pytest

from test_gpu_int_products import _matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["normal", "zeros", "extreme"])
@pytest.mark.parametrize("shape", [(11201, 16, 17), (11101, 16, 33), (11501, 31, 16), (11001, 31, 15), (601, 595, 31),
                                   (600, 587, 31), (6501, 55, 5), (19456, 63, 3), (19457, 63, 3), (1300, 1203, 18),
                                   (38900, 16, 9), (39000, 13, 9)])
def test_bits(T, shape, kind):
    M, N, K = shape
    rng = np.random.default_rng(M + N + K)
    A, B = _matrix(kind, M, K, rng), _matrix(kind, K, N, rng)
    want = np.zeros((M, N))
    with np.errstate(over="ignore", invalid="ignore"):
        for k in range(K):
            want = want + A[:, k:k + 1] * B[k]
    C, _ = T.matmul(A, B)
    assert np.array_equal(C, want, equal_nan=True)
