"""FP64 products on both sides of the line between one thread per output and tiles,
and the tiles' ragged edges, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zeros", [False, True])
@pytest.mark.parametrize("shape", [(512, 512, 16), (513, 513, 31), (16385, 16, 17), (16383, 17, 48), (8193, 33, 15),
                                   (262145, 1, 5), (1, 262145, 3), (5, 60001, 33), (700, 401, 65)])
def test_bits(T, shape, zeros):
    M, N, K = shape
    rng = np.random.default_rng(M + N + K)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    if zeros:
        A[rng.random(A.shape) < 0.3] = 0.0
        B[:, ::3] = 1.0
    want = np.zeros((M, N))
    for k in range(K):
        want = want + A[:, k:k + 1] * B[k]
    C, _ = T.matmul(A, B)
    assert np.array_equal(C, want)
