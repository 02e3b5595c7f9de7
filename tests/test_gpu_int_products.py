"""rrLU with products and quotients on the integer pipes (ieee_int.h): bits of
the factors against the oracle at the edges of the 16 x 8 update tiles, on
values that take the integer path (zeros of both signs among them) and on
values outside its range, which take the FP64 one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(x):
    return np.ascontiguousarray(x, dtype=np.float64).view(np.int64)


def _same(g, r):
    K = r["npivot"]
    assert g.npivot == K
    assert np.array_equal(g.rowpermutation - 1, r["rowpermutation"])
    assert np.array_equal(g.colpermutation - 1, r["colpermutation"])
    # L's unit diagonal and the zero halves are written by both sides as constants
    assert np.array_equal(_bits(g.L), _bits(r["L"]))
    assert np.array_equal(_bits(g.U), _bits(r["U"]))


def _matrix(kind, m, n, rng):
    A = rng.standard_normal((m, n))
    if kind == "zeros":  # a third of the entries, half of them -0
        z = rng.random((m, n))
        A[z < 0.33] = 0.0
        A[z < 0.16] = -0.0
    if kind == "wide":  # magnitudes from 1e-140 to 1e140
        A *= 10.0 ** rng.uniform(-140, 140, size=(m, n))
    if kind == "extreme":  # some entries outside the integer range, subnormals among them
        z = rng.random((m, n))
        A[z < 0.1] *= 1e-200
        A[z < 0.03] *= 1e-115
        A[z > 0.97] *= 1e155
    if kind == "integers":
        A = rng.integers(-4, 5, size=(m, n)).astype(float)
    return A


@pytest.mark.parametrize("kind", ["normal", "zeros", "wide", "extreme", "integers"])
@pytest.mark.parametrize("shape", [(2, 2), (9, 8), (16, 9), (17, 24), (24, 17), (25, 33), (40, 129), (129, 40),
                                   (96, 97), (181, 175)])
def test_tile_edges(T, oracle, shape, kind):
    rng = np.random.default_rng(shape[0] * 977 + shape[1])
    A = _matrix(kind, *shape, rng)
    for left in (True, False):
        try:
            r = oracle.rrlu(A, leftorthogonal=left)
        except oracle.OracleError:
            with pytest.raises(T.TCIError):
                T.rrlu(A, leftorthogonal=left)
            continue
        _same(T.rrlu(A, leftorthogonal=left), r)


@pytest.mark.parametrize("kind", ["normal", "zeros", "wide", "extreme"])
def test_multi_cta(T, oracle, kind):
    A = _matrix(kind, 530, 517, np.random.default_rng(3))
    for left in (True, False):
        _same(T.rrlu(A, leftorthogonal=left, maxrank=70), oracle.rrlu(A, leftorthogonal=left, maxrank=70))
