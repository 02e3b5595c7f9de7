"""L and U of rrlu on both sides of the size up to which the host forms them, for
either side's unit diagonal, capped ranks and results that are not asked for."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left", [True, False])
@pytest.mark.parametrize("maxrank", [1, 7, None])
@pytest.mark.parametrize("shape", [(1, 1), (1, 9), (9, 1), (5, 40), (128, 256), (257, 128), (129, 255), (4, 8192),
                                   (8193, 4)])
def test_bits(T, oracle, shape, maxrank, left):
    a = np.random.default_rng(shape[0]).standard_normal(shape)
    g = T.rrlu(a, maxrank=maxrank, leftorthogonal=left)
    r = oracle.rrlu(a, maxrank=maxrank, leftorthogonal=left)
    assert g.npivot == r["npivot"] and g.error == r["error"]
    for name in ("L", "U"):
        assert np.array_equal(getattr(g, name), r[name])


@pytest.mark.parametrize("shape", [(20, 30), (200, 300)])
def test_only_what_is_asked_for(T, shape):
    m, n = shape
    k = min(shape)
    a = np.asfortranarray(np.random.default_rng(2).standard_normal(shape))
    want = T.rrlu(a)
    lib, ctx = T.load_library(), T.default_context()

    def p(x, t=ctypes.c_double):
        return None if x is None else x.ctypes.data_as(ctypes.POINTER(t))

    for have_l, have_u in ((True, False), (False, True), (False, False)):
        L = np.zeros((m, k), order="F") if have_l else None
        U = np.zeros((k, n), order="F") if have_u else None
        rp, cp = np.zeros(m, np.int64), np.zeros(n, np.int64)
        K, err = ctypes.c_int64(), ctypes.c_double()
        assert lib.tci_rrlu(ctx.h, p(a), m, n, 0, 1e-14, 0.0, 1, p(rp, ctypes.c_int64), p(cp, ctypes.c_int64), p(L),
                            p(U), ctypes.byref(K), ctypes.byref(err)) == 0
        assert K.value == want.npivot and np.array_equal(rp, want.rowpermutation)
        assert np.array_equal(cp, want.colpermutation)
        assert L is None or np.array_equal(L, want.L)
        assert U is None or np.array_equal(U, want.U)
