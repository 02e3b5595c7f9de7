"""A context lives as long as anything that came from it: a garbage collector
finalizes a context and the solves, trains and buffers that refer to it in any order,
at the end of the interpreter above all."""
import gc
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _solve(T, ctx, n=4):
    return T.crossinterpolate2(float, T.DeviceFunction("lorentz"), [n] * 5, tolerance=1e-8, ctx=ctx)[0]


def test_solves_and_buffers_after_the_context_handle(T):
    ctx = T.Context(0)
    tcis = [_solve(T, ctx, n) for n in (4, 5, 6)]
    want = [t.sitetensors() if callable(t.sitetensors) else t.sitetensors for t in tcis]
    values = [t.evaluate([[2] * 5, [3] * 5]) for t in tcis]
    trains = T.tensortrains(tcis, ctx=ctx)
    srv_ctx = T.Context(0)
    srv = T.Server(max_live=4, ctx=srv_ctx)
    srv_ctx.close()
    rid = srv.submit(T.DeviceFunction("lorentz"), [4] * 4, tolerance=1e-6)
    got = []
    while not got:
        got = srv.poll(timeout_ms=100)
    srv.stop()
    assert got[0][0] == rid and got[0][1] == 0
    ctx.close()
    for t, v in zip(tcis, values):
        assert np.array_equal(t.evaluate([[2] * 5, [3] * 5]), v)
    del tcis[1:], t
    gc.collect()
    assert np.array_equal(tcis[0].evaluate([[2] * 5, [3] * 5]), values[0])
    del tcis
    gc.collect()
    for tt, w in zip(trains, want):  # pinned memory of the context
        for a, b in zip(tt.sitetensors, w):
            assert np.array_equal(a, b)


def test_cycles_and_the_end_of_the_interpreter(T):
    code = """
import gc, sys
sys.path.insert(0, %r)
import tci_gb300 as T
class Node: pass
def make():
    n = Node(); n.me = n
    n.ctx = T.Context(0)
    n.f = T.BatchFunction(lambda p: 1.0 / (1.0 + (p * p).sum(1)))
    n.solves = [T.crossinterpolate2(float, f, [4] * 4, tolerance=1e-6, ctx=n.ctx)[0]
                for f in (n.f, T.DeviceFunction("lorentz")) for _ in range(5)]
    n.trains = T.tensortrains(n.solves, ctx=n.ctx)
    return n
for _ in range(3):
    n = make()
    del n
    gc.collect()
keep = [make() for _ in range(2)]
keep.append(keep)
other = T.crossinterpolate2(float, T.DeviceFunction("lorentz"), [4] * 4, tolerance=1e-6)[0]
g = lambda: other
print("end", flush=True)
""" % os.path.join(ROOT, "tensorcrossinterpolation.jl_gb300")
    env = dict(os.environ, MALLOC_PERTURB_="165")  # freed memory is overwritten
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120, env=env)
    assert r.returncode == 0 and r.stdout.strip() == "end", (r.returncode, r.stderr[-2000:])
