"""Performance cases of the TCI2 library: the calls its users make, through the
public Python package and C ABI, over the range of sizes, shapes and options
those calls take.

listed() names fixed cases, draw() gives further ones of the same ranges,
prepare() makes what a program holds before the call (from the seed alone),
run() is one pass, work() the least traffic and arithmetic of a pass and
exact() what a pass returns in plain 64-bit torch / numpy, where that exists.
"""
import ctypes
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.abspath("."), "tensorcrossinterpolation.jl_gb300"))
import tci_gb300 as T  # noqa: E402
from tci_gb300 import workloads  # noqa: E402


# ----------------------------------------------------------------- the cases
def listed():
    return [
        # a small Pi already on the device, factored in a caller's own allocation-free loop: latency
        {"name": "rrlu_device_24", "kind": "rrlu_device", "m": 24, "n": 24, "maxrank": 24, "rank": 24, "left": True},
        # the Pi of an ordinary bond on caller-owned device buffers, ragged and not square
        {"name": "rrlu_device_381x517", "kind": "rrlu_device", "m": 381, "n": 517, "maxrank": 256, "rank": 140,
         "left": False},
        # one large dense matrix from and to host memory (the 2048 x 2048 benchmark configuration)
        {"name": "rrlu_host_2048", "kind": "rrlu_host", "m": 2048, "n": 2048, "maxrank": 512, "left": True},
        # many ragged Pi matrices in one call (the batched benchmark's sizes, ranks as in a sweep: half of 2r)
        {"name": "rrlu_batched_1000", "kind": "rrlu_batched", "count": 1000, "rmin": 8, "rmax": 128},
        # single solves with a registered f, results brought to the host: low rank (latency of small dependent
        # steps), a long quantics train of 2-valued sites, and a quantics train of rank 80
        {"name": "solve_lorentz_8", "kind": "solve", "f": "lorentz", "L": 8, "d": 10, "tol": 1e-8, "maxbond": 200},
        {"name": "solve_qtt1d_40", "kind": "solve", "f": "qtt1d", "L": 40, "d": 2, "tol": 1e-10, "maxbond": 128},
        {"name": "solve_qtt2d_30", "kind": "solve", "f": "qtt2d", "L": 30, "d": 4, "tol": 1e-9, "maxbond": 512},
        # a solve whose f is the caller's own vectorized Python function
        {"name": "solve_caller_f", "kind": "solve", "f": "caller", "L": 8, "d": 10, "tol": 1e-8, "maxbond": 200},
        # a batch of the served family with every train brought back to the host: throughput
        {"name": "batch_2000", "kind": "batch", "count": 2000},
        # evaluation of a train at many points, FP64 with the bonds of a two-dimensional quantics train
        {"name": "evaluate_fp64", "kind": "evaluate", "L": 30, "d": 4, "r": 80, "points": 100000,
         "precision": "fp64"},
        # ... and in split precision with the small bonds of a one-dimensional one, a million points
        {"name": "evaluate_split", "kind": "evaluate", "L": 40, "d": 2, "r": 12, "points": 1000000,
         "precision": "tf32x3"},
        # an operator applied to a train by zip-up, FP64
        {"name": "contract_zipup", "kind": "contract", "L": 16, "d": 4, "ra": 24, "rb": 60, "maxbond": 200,
         "tol": 1e-9, "method": "LU", "precision": "fp64"},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["rrlu_device", "rrlu_device", "rrlu_host", "rrlu_batched", "solve", "solve", "batch",
                       "evaluate", "evaluate", "contract"])
    if kind == "rrlu_device":
        m = _log(rng, 5, 1000)
        n = min(_log(rng, 5, 1000), 524288 // m)
        k = min(m, n)
        return {"kind": kind, "m": m, "n": n, "maxrank": rng.randint(max(1, k // 2), k),
                "rank": rng.randint(max(1, k // 3), k), "left": rng.random() < 0.5}
    if kind == "rrlu_host":
        m, n = _log(rng, 60, 2048), _log(rng, 60, 2048)
        return {"kind": kind, "m": m, "n": n, "maxrank": min(512, _log(rng, 20, min(m, n))), "left": rng.random() < 0.5}
    if kind == "rrlu_batched":
        rmax = rng.randint(16, 128)
        return {"kind": kind, "count": _log(rng, 50, 1000), "rmin": rng.randint(4, rmax), "rmax": rmax}
    if kind == "solve":
        f = rng.choice(["lorentz", "served", "qtt1d", "qtt2d", "caller"])
        tol = float("%.1e" % 10 ** rng.uniform(-10, -6))
        if f in ("lorentz", "caller"):
            return {"kind": kind, "f": f, "L": rng.randint(4, 9), "d": rng.randint(3, 11), "tol": tol, "maxbond": 200}
        if f == "served":
            return {"kind": kind, "f": f, "L": rng.randint(4, 16), "d": rng.randint(2, 16), "tol": tol,
                    "maxbond": rng.choice([32, 64, 128])}
        if f == "qtt1d":
            return {"kind": kind, "f": f, "L": rng.randint(16, 40), "d": 2, "tol": tol, "maxbond": 128}
        return {"kind": kind, "f": f, "L": rng.randint(14, 30), "d": 4, "tol": max(tol, 1e-9), "maxbond": 512}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 30, 2000)}
    if kind == "evaluate":
        if rng.random() < 0.5:
            return {"kind": kind, "L": rng.randint(4, 40), "d": rng.randint(2, 5), "r": rng.randint(17, 90),
                    "points": _log(rng, 50, 60000), "precision": rng.choice(["fp64", "tf32x3"])}
        return {"kind": kind, "L": rng.randint(4, 40), "d": rng.randint(2, 16), "r": rng.randint(2, 16),
                "points": _log(rng, 50, 1000000), "precision": rng.choice(["fp64", "tf32x3"])}
    return {"kind": kind, "L": rng.randint(4, 16), "d": rng.randint(2, 4), "ra": _log(rng, 2, 24),
            "rb": _log(rng, 6, 60), "maxbond": rng.randint(16, 200), "tol": 1e-9,
            "method": rng.choice(["LU", "LU", "CI"]), "precision": rng.choice(["fp64", "fp64", "tf32x3"])}


# -------------------------------------------------------------------- inputs
def _train(case, rng, r, d, legs, L):
    """Cores of a random train whose values stay of order one: bonds up to r,
    smaller at the ends where prod(d) does not allow r."""
    q = d ** legs
    bonds = [1] + [min(r, q ** min(b, L - b, 12)) for b in range(1, L)] + [1]
    shape = (d,) * legs
    return [rng.standard_normal((bonds[b],) + shape + (bonds[b + 1],)) / np.sqrt(bonds[b]) for b in range(L)]


def _graded(rng, m, n, rank):
    """An m x n matrix whose singular values fall to 1e-10 at about `rank`, plus noise."""
    k = min(m, n, rank + rank // 5 + 1)
    s = 10.0 ** (-10.0 * np.arange(k) / max(rank, 1))
    return (rng.standard_normal((m, k)) * s) @ rng.standard_normal((k, n)) / k + 1e-14 * rng.standard_normal((m, n))


def _sizes(case):
    """Row counts of a batch of matrices: part of the case, not of the seed."""
    rng = np.random.default_rng([case["count"], case["rmin"], case["rmax"]])
    return [2 * int(rng.integers(case["rmin"], case["rmax"] + 1)) for _ in range(case["count"])]


# Room for the site tensors of one solve in a program's own result buffer, in doubles.
ROOM = {"lorentz": 60000, "caller": 60000, "served": 200000, "qtt1d": 100000, "qtt2d": 1500000}


def _first_pivot(case, rng):
    """A start point where f is not negligible."""
    L = case["L"]
    if case["f"] == "qtt2d":  # near the centre of the Gaussian
        x, y = (int((0.4 + 0.2 * rng.random()) * 2.0 ** L) for _ in range(2))
        return [1 + ((x >> (L - 1 - p)) & 1) + 2 * ((y >> (L - 1 - p)) & 1) for p in range(L)]
    return [int(v) for v in rng.integers(1, case["d"] + 1, size=L)]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    ctx = T.default_context()
    st = {"case": case, "ctx": ctx}
    if kind == "rrlu_device":
        m, n = case["m"], case["n"]
        a = _graded(rng, m, n, case["rank"])
        st["a"] = torch.tensor(np.ascontiguousarray(a.T), dtype=torch.float64, device="cuda")  # column-major m x n
        dev = {"device": "cuda"}
        st["rowperm"] = torch.zeros(m, dtype=torch.int32, **dev)
        st["colperm"] = torch.zeros(n, dtype=torch.int32, **dev)
        st["npivot"] = torch.zeros(1, dtype=torch.int32, **dev)
        st["error"] = torch.zeros(1, dtype=torch.float64, **dev)
        st["status"] = torch.zeros(1, dtype=torch.int32, **dev)
        st["factors"] = torch.zeros((n, m), dtype=torch.float64, **dev)
    elif kind == "rrlu_host":
        st["a"] = np.asfortranarray(rng.standard_normal((case["m"], case["n"])))
    elif kind == "rrlu_batched":
        mats = []
        for n in _sizes(case):
            mats.append(np.asfortranarray(_graded(rng, n, n, n // 2)))
        st["mats"] = mats
        st["rows"] = np.zeros((len(mats), 2 * case["rmax"]), np.int64)
        st["cols"] = np.zeros_like(st["rows"])
    elif kind == "solve":
        L, d = case["L"], case["d"]
        st["dims"] = [d] * L
        st["pivot"] = [_first_pivot(case, rng)]
        st["kw"] = dict(tolerance=case["tol"], maxbonddim=case["maxbond"], maxiter=20, seed=int(seed) & 0xffff)
        if case["f"] == "lorentz":
            st["f"] = T.DeviceFunction("lorentz", [1.0 + rng.random()])
        elif case["f"] == "served":
            a, b, g = 10 ** rng.uniform(-2, 1, size=3)
            c = rng.integers(1, d + 1, size=L)
            st["f"] = T.DeviceFunction("served", [a, b, g] + [float(x) for x in c])
        elif case["f"] == "caller":
            scale = 1.0 + rng.random()
            st["f"] = T.BatchFunction(lambda p: scale / (1.0 + (p * p).sum(1)))
        else:
            st["f"] = T.DeviceFunction(case["f"], [0] if case["f"] == "qtt1d" else [])
        st["cores"] = np.zeros(ROOM[case["f"]])
    elif kind == "batch":
        reqs = workloads.served_requests(case["count"], int(seed))
        st["specs"] = [(T.DeviceFunction("served", p), [d] * L, dict(tolerance=tol, maxbonddim=mbd))
                       for L, d, p, tol, mbd in reqs]
        st["cores"] = np.zeros(12000 * case["count"] + 400000)  # about 9000 doubles a solve on average
    elif kind == "evaluate":
        st["tt"] = T.TensorTrain(_train(case, rng, case["r"], case["d"], 1, case["L"]))
        st["points"] = rng.integers(1, case["d"] + 1, size=(case["points"], case["L"]))
    else:
        st["a"] = _train(case, rng, case["ra"], case["d"], 2, case["L"])
        st["b"] = T.TensorTrain(_train(case, rng, case["rb"], case["d"], 1, case["L"]))
    return st


# -------------------------------------------------------------------- a pass
def _fetch(tcis, out, max_sites, ctx):
    """Every site tensor of the solves into the program's own buffer; returns all their shapes."""
    lib = T.load_library()
    n = len(tcis)
    handles = (ctypes.c_void_p * n)(*[t.h.value for t in tcis])
    lens = np.array([len(t) for t in tcis])
    dims = np.zeros((max_sites * n, 3), np.int64)  # the sites of all solves in a row, then zeros
    i64p, f64p = ctypes.POINTER(ctypes.c_int64), ctypes.POINTER(ctypes.c_double)
    rc = lib.tci_get_core_dims_batched(n, handles, dims.ctypes.data_as(i64p))
    ends = np.cumsum(dims.prod(axis=1))[np.cumsum(lens) - 1]
    if rc or ends[-1] > out.size:
        raise RuntimeError(f"site tensors: code {rc}, {ends[-1]} values for a buffer of {out.size}")
    offs = np.ascontiguousarray(np.concatenate([[0], ends[:-1]]), dtype=np.int64)
    rc = lib.tci_get_cores_batched(ctx.h, n, handles, out.ctypes.data_as(f64p), offs.ctypes.data_as(i64p))
    if rc:
        raise RuntimeError(f"site tensors: code {rc}")
    return dims


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "rrlu_device":
        def p(t):
            return ctypes.c_void_p(t.data_ptr())
        rc = T.load_library().tci_rrlu_noalloc(
            p(st["a"]), case["m"], case["n"], case["maxrank"], 1e-10, 0.0, int(case["left"]), p(st["rowperm"]),
            p(st["colperm"]), p(st["npivot"]), p(st["error"]), p(st["status"]), p(st["factors"]),
            torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError(f"tci_rrlu_noalloc: {rc}")
        return {k: st[k] for k in ("rowperm", "colperm", "npivot", "error", "status", "factors")}
    if kind == "rrlu_host":
        r = T.rrlu(st["a"], maxrank=case["maxrank"], reltol=1e-10, leftorthogonal=case["left"], ctx=ctx)
        return {"rowperm": r.rowpermutation, "colperm": r.colpermutation, "L": r.L, "U": r.U, "npivot": r.npivot,
                "error": r.error}
    if kind == "rrlu_batched":
        out = T.rrlu_batched(st["mats"], maxrank=256, reltol=1e-10, ctx=ctx)
        for i, (rows, cols, k, _) in enumerate(out):
            st["rows"][i, :k] = rows
            st["cols"][i, :k] = cols
        return {"rows": st["rows"], "cols": st["cols"], "npivot": np.array([o[2] for o in out]),
                "error": np.array([o[3] for o in out])}
    if kind == "solve":
        tci, ranks, errors = T.crossinterpolate2(float, st["f"], st["dims"], st["pivot"], ctx=ctx, **st["kw"])
        bonds = _fetch([tci], st["cores"], case["L"], ctx)
        return {"cores": st["cores"], "bonds": bonds, "rank": int(ranks[-1]), "error": float(errors[-1])}
    if kind == "batch":
        tcis = T.crossinterpolate2_batched(st["specs"], max_live=1024, ctx=ctx)
        return {"cores": st["cores"], "bonds": _fetch(tcis, st["cores"], 16, ctx)}
    if kind == "evaluate":
        return st["tt"].evaluate(st["points"], ctx=ctx, precision=case["precision"])
    res = T.contract(st["a"], st["b"], algorithm="zipup", tolerance=case["tol"], maxbonddim=case["maxbond"],
                     method=case["method"], ctx=ctx, precision=case["precision"])
    return res.sitetensors


# ---------------------------------------------------------------- least work
def _lu_work(m, n, k):
    flops = 2.0 * sum((m - q) * (n - q) for q in range(1, k))
    return flops


def work(case):
    kind = case["kind"]
    if kind in ("rrlu_device", "rrlu_host"):
        m, n = case["m"], case["n"]
        k = min(m, n, case["maxrank"], case.get("rank", m))
        out = m * n if kind == "rrlu_device" else (m + n) * k
        return {"bytes": 8.0 * (m * n + out) + 8.0 * (m + n), "flops": _lu_work(m, n, k)}
    if kind == "rrlu_batched":
        rs = np.linspace(case["rmin"], case["rmax"], 9)
        per = np.mean([_lu_work(int(2 * r), int(2 * r), int(r)) for r in rs])
        size = np.mean([4 * r * r + 2 * r for r in rs])
        return {"bytes": 8.0 * case["count"] * size, "flops": case["count"] * per}
    if kind == "solve":
        # nominal: three iterations of two half sweeps at the rank such an f has, with a rank-r LU of an
        # (r d) x (r d) Pi per bond
        r = {"lorentz": 12, "caller": 12, "served": 20, "qtt1d": 11, "qtt2d": 80}[case["f"]]
        L, d = case["L"], case["d"]
        m = r * d
        return {"bytes": 8.0 * L * d * r * r, "flops": 6.0 * L * (_lu_work(m, m, r) / 4 + 2 * m * r * r)}
    if kind == "batch":  # means of the family: 10 sites of 9 values, rank 20
        per = 6.0 * 10 * (_lu_work(180, 180, 20) / 4 + 2 * 180 * 400)
        return {"bytes": 8.0 * case["count"] * 10 * 9 * 400, "flops": case["count"] * per}
    L, d = case["L"], case["d"]
    if kind == "evaluate":
        q = [min(case["r"], d ** min(b, L - b, 12)) for b in range(L + 1)]
        q[0] = q[L] = 1
        per = 2.0 * sum(q[b] * q[b + 1] for b in range(L))
        size = sum(q[b] * d * q[b + 1] for b in range(L))
        return {"bytes": 8.0 * (size + case["points"]) + case["points"] * L, "flops": per * case["points"]}
    ra, rb, k = case["ra"], case["rb"], case["maxbond"]
    per = 2.0 * k * rb * d * d * ra * ra + 2.0 * k * d * ra * rb * d * rb + _lu_work(k * d, ra * rb, min(k, ra * rb))
    return {"bytes": 8.0 * L * (ra * ra * d * d + rb * rb * d + k * k * d), "flops": per * max(1, L - 4)}


# ------------------------------------------------------------ 64-bit results
def _rrlu(a, maxrank, reltol, left):
    """Full-pivot rank-revealing LU in plain torch (float64)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    A = torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    m, n = A.shape
    rp, cp = np.arange(m), np.arange(n)
    maxerr, err, K = 0.0, float("nan"), 0
    while K < min(maxrank, m, n):
        sub = A[K:, K:].t().contiguous()  # ties go to the first element in column-major order
        pos = int(torch.argmax(sub * sub))
        r, c = K + pos % (m - K), K + pos // (m - K)
        piv = float(A[r, c])
        err = abs(piv)
        if K > 0 and err < reltol * maxerr:
            break
        maxerr = max(maxerr, err)
        if r != K:
            A[[K, r]] = A[[r, K]]
            rp[[K, r]] = rp[[r, K]]
        if c != K:
            A[:, [K, c]] = A[:, [c, K]]
            cp[[K, c]] = cp[[c, K]]
        if left:
            A[K + 1:, K] /= piv
        else:
            A[K, K + 1:] /= piv
        K += 1
        if K < min(maxrank, m, n):
            A[K:, K:] -= torch.outer(A[K:, K - 1], A[K - 1, K:])
    if K >= min(m, n):
        err = 0.0
    return A.cpu().numpy(), rp, cp, K, err


def exact(case, seed):
    kind = case["kind"]
    if kind == "evaluate":
        st = prepare(case, seed)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        pts = torch.tensor(st["points"] - 1, device=dev)
        v = torch.ones((pts.shape[0], 1), dtype=torch.float64, device=dev)
        for b, core in enumerate(st["tt"].sitetensors):
            c = torch.tensor(np.ascontiguousarray(core), device=dev)
            w = torch.empty((pts.shape[0], c.shape[2]), dtype=torch.float64, device=dev)
            for i in range(c.shape[1]):
                sel = pts[:, b] == i
                w[sel] = v[sel] @ c[:, i, :]
            v = w
        return v[:, 0].cpu().numpy()
    if kind in ("rrlu_device", "rrlu_host"):
        st = prepare(case, seed)
        a = st["a"].cpu().numpy().T if kind == "rrlu_device" else st["a"]
        A, rp, cp, K, err = _rrlu(a, case["maxrank"], 1e-10, case["left"])
        if kind == "rrlu_device":
            return {"rowperm": None, "colperm": None, "npivot": None, "error": err, "status": None, "factors": A.T}
        Lm, U = np.tril(A[:, :K]), np.triu(A[:K, :])
        np.fill_diagonal(Lm if case["left"] else U, 1.0)
        return {"rowperm": None, "colperm": None, "L": Lm, "U": U, "npivot": None, "error": err}
    if kind == "rrlu_batched" and case["count"] * case["rmax"] <= 20000:
        errs = [_rrlu(a, 256, 1e-10, True)[4] for a in prepare(case, seed)["mats"]]
        return {"rows": None, "cols": None, "npivot": None, "error": np.array(errs)}
    return None  # a solve or a truncated contraction: its values depend on the pivots it takes
