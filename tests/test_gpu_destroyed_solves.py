"""Solves destroyed while another thread holds their context are released by that
thread: the device memory of a caller-supplied f's value cache (a CUDA allocation of
its own) is free again once the server that held the context has stopped, with no
further call on the context."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_memory_of_solves_destroyed_under_a_server(T):
    torch = pytest.importorskip("torch")
    ctx = T.Context(0)
    f = T.BatchFunction(lambda p: 1.0 / (1.0 + (p * p).sum(1)))
    old = [T.crossinterpolate2(float, f, [10] * 8, tolerance=1e-8, ctx=ctx)[0] for _ in range(8)]
    entries = sum(s.fcache_stats()[0] for s in old)
    reg = T.DeviceFunction("lorentz")
    plain = [T.crossinterpolate2(float, reg, [4] * 4, tolerance=1e-6, ctx=ctx)[0] for _ in range(3)]
    srv = T.Server(max_live=4, ctx=ctx)
    srv.submit(reg, [4] * 4, tolerance=1e-6)
    got = []
    while not got:  # from here on the server holds the context and waits for requests
        got = srv.poll(timeout_ms=100)
    assert got[0][1] == 0
    before = torch.cuda.mem_get_info(0)[0]

    def drop():
        old.clear()
        plain.clear()

    th = threading.Thread(target=drop)
    th.start()
    th.join(20)
    assert not th.is_alive()
    srv.stop()
    # a cache entry is 32 bytes and at most half of a table is in use
    assert entries > 100000
    assert torch.cuda.mem_get_info(0)[0] - before >= 64 * entries
