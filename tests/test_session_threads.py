"""Threads that share one session: no call may read or write through the addresses of another."""
import ctypes
import threading
from types import SimpleNamespace

import numpy as np
import pytest

from oxionnx_b200 import _ffi, models
from oxionnx_b200 import session as S
from oxionnx_b200.graph import Graph


class _Library:
    """Stands in for the C library: y = x + 1 over three lanes.  Every call first waits a moment for another thread to
    come as far, which only happens when the callers do not keep out of one another's way."""

    def __init__(self):
        self.inside, self.meeting = 0, threading.Event()

    def oxb200_fetch_value(self, handle, name, result):
        r = result._obj
        r.rank, r.len, r.shape[0] = 1, 3, 3
        return _ffi.OK_HOST

    def oxb200_last_error(self, handle):
        return b""

    def oxb200_run(self, handle, feeds, n_in, fetches, n_out):
        self.inside += 1
        if self.inside == 2:
            self.meeting.set()
        self.meeting.wait(0.3)
        x = np.ctypeslib.as_array(feeds[0].lanes, (3,))
        ctypes.memmove(fetches[0].lanes, (x + 1).ctypes.data, 12)
        return _ffi.OK_HOST

    def oxb200_run_bound(self, handle, feeds, n_in, fetches, n_out):
        return self.oxb200_run(handle, feeds, n_in, fetches, n_out)


def _in_threads(calls):
    outs = [None] * len(calls)

    def work(i):
        outs[i] = calls[i]()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return outs


@pytest.mark.parametrize("entry", ["run", "run_with_binding"])
def test_calls_of_two_threads_keep_their_own_buffers(monkeypatch, entry):
    library = _Library()
    monkeypatch.setattr(_ffi, "lib", lambda: library)
    monkeypatch.setattr(S, "CudaContext", lambda device, **kw: SimpleNamespace(handle=None, register_weights=lambda w: None, last_error=lambda: ""))
    session = S.Session(Graph(nodes=[], input_names=["x"], output_names=["y"]), {}, 0, {}, {})
    session._planned_for = {"x": (3,)}
    feeds = [np.float32([1, 2, 3]), np.float32([10, 20, 30])]  # held here, so a mixed-up address is still one that may be read
    outs = _in_threads([lambda f=f: getattr(session, entry)({"x": f}) for f in feeds])
    for f, out in zip(feeds, outs):
        assert np.array_equal(out["y"], f + 1)


@pytest.mark.gpu
def test_threads_share_a_planned_session():
    graph, weights, feeds, _ = models.build_int8_mlp(rows=8, dims=(128, 256, 128), spelling="qlinearmatmul")
    session = S.Session.builder().build_from_graph(graph, weights)
    base = feeds()["x"]
    batches = [np.roll(base, i, axis=0) * np.float32(1 + 0.1 * i) for i in range(8)]
    # every other batch has another number of rows, so the threads also plan in turn
    batches = [b if i % 4 else b[:5] for i, b in enumerate(batches)]
    want = [session.run({"x": b})["y"].copy() for b in batches]

    def many(b):
        return [session.run({"x": b.astype(np.float64)})["y"] for _ in range(20)]

    for got, w in zip(_in_threads([lambda b=b: many(b) for b in batches]), want):
        assert all(np.array_equal(g, w) for g in got)
    session.close()


@pytest.mark.gpu
def test_messages_of_failing_threads_are_whole():
    """Threads that share a context and are refused all the time: every message read is one that some call left."""
    ctx = S.CudaContext(0)
    lib = _ffi.lib()
    expected = {f"attribute '{c * 60}' has a kind this provider does not handle" for c in "abcd"}

    def refused(letter):
        attr = (_ffi.Attr * 1)()
        attr[0].name, attr[0].kind = (letter * 60).encode(), 99
        node, keep = _ffi.CNode(), _ffi.Keep()
        node.op_type, node.attrs, node.n_attrs = b"Relu", attr, 1
        results = (_ffi.Result * 1)()
        seen = set()
        for _ in range(2000):
            assert lib.oxb200_dispatch(ctx.handle, ctypes.byref(node), None, 0, 0, results, 0) == _ffi.DECLINED
            seen.add(ctx.last_error())
        return seen

    for seen in _in_threads([lambda c=c: refused(c) for c in "abcd"]):
        assert seen <= expected
    assert ctx.cache_counters()["declines"] == 8000
    ctx.close()
