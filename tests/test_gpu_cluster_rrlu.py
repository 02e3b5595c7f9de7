"""tci_rrlu_noalloc on thread-block clusters: bits against the oracle at the
sizes where its block grid, its tiles and the rule that picks it change."""
import ctypes

import numpy as np
import pytest

from test_gpu_int_products import _bits, _matrix

pytestmark = pytest.mark.gpu


def _rrlu(T, A, maxrank, left, reltol=1e-14, factors=True):
    import torch

    m, n = A.shape
    dev = {"device": "cuda"}
    a = torch.tensor(np.ascontiguousarray(A.T), **dev)
    rp, cp = torch.zeros(m, dtype=torch.int32, **dev), torch.zeros(n, dtype=torch.int32, **dev)
    k, st = torch.zeros(1, dtype=torch.int32, **dev), torch.full((1,), -1, dtype=torch.int32, **dev)
    err, fact = torch.zeros(1, dtype=torch.float64, **dev), torch.zeros((n, m), dtype=torch.float64, **dev)

    def p(t):
        return ctypes.c_void_p(t.data_ptr())

    rc = T.load_library().tci_rrlu_noalloc(p(a), m, n, maxrank, reltol, 0.0, int(left), p(rp), p(cp), p(k), p(err),
                                           p(st), p(fact) if factors else None,
                                           torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return (rp.cpu().numpy(), cp.cpu().numpy(), int(k), float(err), int(st), fact.cpu().numpy().T,
            np.array_equal(a.cpu().numpy().T, A, equal_nan=True))


def _check(T, oracle, A, maxrank=0, left=True, **kw):
    rp, cp, K, err, st, F, kept = _rrlu(T, A, maxrank, left, **kw)
    assert kept
    r = oracle.rrlu(A, leftorthogonal=left, **({"maxrank": maxrank} if maxrank else {}), **kw)
    assert (st, K) == (0, r["npivot"])
    assert np.array_equal(rp, r["rowpermutation"]) and np.array_equal(cp, r["colpermutation"])
    assert err == r["error"] or (np.isnan(err) and np.isnan(r["error"]))
    L, U = np.tril(F[:, :K]), np.triu(F[:K, :])
    np.fill_diagonal(L if left else U, 1.0)
    assert np.array_equal(_bits(L), _bits(r["L"])) and np.array_equal(_bits(U), _bits(r["U"]))


@pytest.mark.parametrize("kind", ["normal", "zeros", "wide", "extreme", "integers"])
@pytest.mark.parametrize("shape", [(32, 33), (49, 51), (50, 50), (100, 100), (5, 600), (601, 5), (67, 129), (190, 65), (250, 243)])
def test_shapes(T, oracle, shape, kind):
    A = _matrix(kind, *shape, np.random.default_rng(shape[0] + 7 * shape[1]))
    for left in (True, False):
        try:
            oracle.rrlu(A, leftorthogonal=left)
        except oracle.OracleError:
            assert _rrlu(T, A, 0, left)[4] == T.TCI_ERR_NAN
            continue
        _check(T, oracle, A, left=left)


@pytest.mark.parametrize("shape", [(381, 517), (724, 724), (600, 700), (1, 2000), (16384, 32), (40, 12000)])
def test_large(T, oracle, shape):
    A = np.random.default_rng(5).standard_normal(shape)
    for left in (True, False):
        _check(T, oracle, A, maxrank=40, left=left)


def test_stops_and_nan(T, oracle):
    rng = np.random.default_rng(9)
    A = rng.standard_normal((90, 20)) @ rng.standard_normal((20, 110))
    _check(T, oracle, A, reltol=1e-10)
    _check(T, oracle, A, maxrank=1)
    A[17, 31] = np.nan  # a NaN that joins U or L, and one that stays in the trailing block
    for kw in ({}, {"reltol": 0.0}):
        try:
            oracle.rrlu(A, **kw)
            want = 0
        except oracle.OracleError:
            want = T.TCI_ERR_NAN
        assert _rrlu(T, A, 0, True, **kw)[4] == want
    assert _rrlu(T, np.full((40, 50), np.nan), 0, True)[4] == T.TCI_ERR_NAN
    assert _rrlu(T, A, 3, True)[2] == 3
    got, ref = _rrlu(T, np.nan_to_num(A), 7, False, factors=False), oracle.rrlu(np.nan_to_num(A), maxrank=7,
                                                                              leftorthogonal=False)
    assert got[2] == ref["npivot"] and np.array_equal(got[0], ref["rowpermutation"])
