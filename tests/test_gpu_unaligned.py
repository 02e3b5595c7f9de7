"""Host arrays off their natural alignment (fields of packed records, views into byte
buffers): numpy's ascontiguousarray keeps them so, and a kernel must not read them in
place."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shifted(a, by):
    """The same values in the same order, `by` bytes off alignment."""
    order = "F" if a.flags.f_contiguous else "C"
    buf = np.zeros(a.nbytes + 16, np.uint8)
    lead = -buf.ctypes.data % 8 + by
    out = buf[lead:lead + a.nbytes].view(a.dtype).reshape(a.shape, order=order)
    out[...] = a
    assert out.ctypes.data % 8 == by
    return out


@pytest.mark.parametrize("by", [1, 4])
@pytest.mark.parametrize("precision", ["fp64", "tf32x3"])
@pytest.mark.parametrize("n", [3, 20000])  # eight sites: the device packs from 65536 values on
def test_points(T, by, precision, n):
    rng = np.random.default_rng(n)
    bonds = [1, 2, 4, 8, 16, 8, 4, 2, 1]
    tt = T.TensorTrain([rng.standard_normal((bonds[s], 2, bonds[s + 1])) for s in range(8)])
    pts = rng.integers(1, 3, size=(n, 8))
    off = _shifted(pts, by)
    assert not np.ascontiguousarray(off).flags.aligned
    assert np.array_equal(tt.evaluate(off, precision=precision), tt.evaluate(pts, precision=precision))
    off[n // 2, 3] = 3
    with pytest.raises(T.ArgumentError, match="out of range"):
        tt.evaluate(off, precision=precision)


@pytest.mark.parametrize("shape", [(1, 1), (24, 20), (49, 51), (60, 70), (520, 530)])
def test_rrlu(T, shape):
    a = np.asfortranarray(np.random.default_rng(shape[0]).standard_normal(shape))
    want, got = T.rrlu(a, maxrank=12), T.rrlu(_shifted(a, 4), maxrank=12)
    for name in ("rowpermutation", "colpermutation", "L", "U", "npivot", "error"):
        assert np.array_equal(getattr(got, name), getattr(want, name))


def test_rrlu_batched_of_a_packed_buffer(T):
    rng = np.random.default_rng(3)
    mats = [np.asfortranarray(rng.standard_normal((5 + k, 30 - k))) for k in range(12)]
    want = T.rrlu_batched(mats, maxrank=9)
    flat = _shifted(np.concatenate([a.reshape(-1, order="F") for a in mats]), 4)
    ms = np.array([a.shape[0] for a in mats], np.int64)
    ns = np.array([a.shape[1] for a in mats], np.int64)
    offs = np.concatenate([[0], np.cumsum(ms * ns)[:-1]]).astype(np.int64)
    poffs = 18 * np.arange(len(mats), dtype=np.int64)
    piv, npiv, errs = np.zeros(18 * len(mats), np.int64), np.zeros(len(mats), np.int64), np.zeros(len(mats))

    def p(a, t):
        return a.ctypes.data_as(ctypes.POINTER(t))

    i64, f64 = ctypes.c_int64, ctypes.c_double
    rc = T.load_library().tci_rrlu_batched(T.default_context().h, len(mats), p(flat, f64), p(offs, i64), p(ms, i64),
                                           p(ns, i64), 9, 1e-14, 0.0, 1, p(piv, i64), p(poffs, i64), p(npiv, i64),
                                           p(errs, f64))
    assert rc == 0
    for k, (rows, cols, K, err) in enumerate(want):
        assert npiv[k] == K and errs[k] == err
        assert np.array_equal(piv[poffs[k]:poffs[k] + K], rows)
        first = poffs[k] + min(9, ms[k], ns[k])  # the columns follow the rows' capacity
        assert np.array_equal(piv[first:first + K], cols)
