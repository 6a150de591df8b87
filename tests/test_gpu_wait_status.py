"""Whom a give-up of a bounded wait is reported to: the next call on the same
stream or of the same batch, while calls on other streams run as if nothing
had happened.

The give-up is made to happen with ``sb_debug_wait_limit(0)``; nothing faults
or hangs (see test_gpu_bounded_wait.py)."""

from __future__ import annotations

import ctypes
import time

import numpy as np
import pytest

from stencil_benchmarks_gb300 import _native, kernels
from stencil_benchmarks_gb300.batching import Batch, VadvDomain
from stencil_benchmarks_gb300.device import Event, Field, Stream
from tests.gpu_helpers import VADV_ARGS, VADV_DISTS, bits_equal, download_like, host_field, interior, rng_fields, to_device

pytestmark = pytest.mark.gpu

DOMAIN, HALO = (64, 6, 24), (1, 1, 0)


class _Solve:
    def __init__(self, storage):
        shape = tuple(d + 2 * h for d, h in zip(DOMAIN, HALO))
        hosts = [host_field(v, storage, halo=HALO) for v in rng_fields(1, shape, VADV_ARGS, VADV_DISTS).values()]
        self.like = hosts[0]
        self.fields = [to_device(h, storage, HALO) for h in hosts]
        self.out = Field.like_host(self.like, storage, HALO)
        self.launch()
        _native.synchronize()
        self.want = self.got()
        self.out.upload(np.zeros_like(self.like))

    def launch(self, stream=None):
        kernels.vadv(*self.fields, (1, 0), out=self.out, stream=stream)

    def got(self):
        return interior(download_like(self.out, self.like), DOMAIN, HALO)


def _finish(stream):
    """Wait for the stream without a call that reports give-ups."""
    done = Event()
    done.record(stream)
    deadline = time.monotonic() + 30.0
    while _native.lib().sb_event_query(ctypes.c_void_p(done.handle)) != _native.SB_OK:
        assert time.monotonic() < deadline, "launch did not complete"


@pytest.fixture
def wait_limit(lib):
    yield lambda polls: _native.call("sb_debug_wait_limit", polls)
    _native.call("sb_debug_wait_limit", -1)
    _native.lib().sb_synchronize()


def _reports(call):
    with pytest.raises(_native.SbError) as err:
        call()
    assert err.value.code == _native.SB_ERR_TIMEOUT


@pytest.mark.parametrize("storage", ["float64", "float32"])
def test_other_streams_are_not_affected(storage, wait_limit):
    mine, other = _Solve("float32"), _Solve(storage)
    a, b = Stream(), Stream()
    wait_limit(0)
    mine.launch(a)
    _finish(a)
    wait_limit(-1)
    other.launch(b)  # runs, and says nothing of a's launch
    _finish(b)
    assert bits_equal(other.got(), other.want)
    _reports(lambda: mine.launch(a))
    mine.launch(a)
    a.synchronize()
    assert bits_equal(mine.got(), mine.want)


def test_batches(wait_limit):
    solve, other = _Solve("float32"), _Solve("float64")
    batches = [Batch("float32", max_domains=2, max_nk=32) for _ in range(2)]
    for batch in batches:
        batch.set([VadvDomain(*solve.fields, out=solve.out)])
    a, b = Stream(), Stream()
    wait_limit(0)
    batches[0].launch(a)
    _finish(a)
    wait_limit(-1)
    other.launch(b)
    batches[1].launch(b)
    _finish(b)
    assert bits_equal(other.got(), other.want) and bits_equal(solve.got(), solve.want)
    _reports(lambda: batches[0].launch(b))  # the same batch, wherever it goes next
    wait_limit(0)
    batches[0].launch(a)
    _finish(a)
    wait_limit(-1)
    _reports(lambda: other.launch(a))  # the same stream
    batches[0].launch(a)
    a.synchronize()


def test_synchronising_reports_every_stream(wait_limit):
    solve = _Solve("float32")
    a, b = Stream(), Stream()
    batch = Batch("float32", max_domains=2, max_nk=32)
    batch.set([VadvDomain(*solve.fields, out=solve.out)])
    for launch in (solve.launch, batch.launch):
        for sync in (b.synchronize, lambda: _native.call("sb_synchronize")):
            wait_limit(0)
            launch(a)
            _finish(a)
            _reports(sync)
            sync()  # cleared
    # a batch that ends and a stream that is destroyed before anyone asked
    launch(a)
    _finish(a)
    batch.close()
    _reports(b.synchronize)
    c = Stream()
    solve.launch(c)
    _finish(c)
    c._finalizer()
    _reports(b.synchronize)
    b.synchronize()
