"""The buffers of a served job live until it is waited for or the server is closed.

The library's worker reads a job's raster and writes its results while the job is in
flight, also after the caller has dropped the ticket.  A fake library stands in for it.
"""
import gc
import weakref

import numpy as np
import pytest


class FakeLibrary:
    """Takes every job and leaves it in flight."""

    def __init__(self):
        self.jobs = 0
        self.at_destroy = None
        self.watch = []

    def siting_server_submit(self, h, p, dem, pitch, obs, sel, ticket):
        self.jobs += 1
        ticket._obj.value = self.jobs
        return 0

    def siting_server_wait(self, h, ticket, timeout, info):
        return 0 if ticket <= self.jobs else 1

    def siting_server_destroy(self, h):
        self.at_destroy = [ref() is not None for ref in self.watch]
        return 0

    def siting_status_string(self, rc):
        return b"status"


@pytest.fixture
def server(native):
    srv = native.Server.__new__(native.Server)
    srv._lib, srv.h, srv._held = FakeLibrary(), 1, {}
    yield srv
    srv.close()


def _submit(native, srv):
    p = native.Params(nrows=64, roi=5, height=3, ntests=4, bw=8, nwanted0=64, intervis=0)
    return srv.submit(p, np.zeros(64 * 64, np.uint16))


def test_buffers_outlive_a_dropped_ticket(native, server):
    t = _submit(native, server)
    server._lib.watch = [weakref.ref(a) for a in (t.dem, t.obs, t.selected)]
    del t
    gc.collect()
    assert all(ref() is not None for ref in server._lib.watch)
    server.close()
    assert server._lib.at_destroy == [True] * 3  # still there when the worker ends
    gc.collect()
    assert all(ref() is None for ref in server._lib.watch)


def test_buffers_go_with_the_ticket_once_waited_for(native, server):
    t = _submit(native, server)
    refs = [weakref.ref(a) for a in (t.dem, t.obs, t.selected)]
    server.wait(t)
    del t
    gc.collect()
    assert all(ref() is None for ref in refs)
