"""A server whose kernels give up a bounded wait: no request with an incomplete
output is reported as completed, none is lost, and all run again, to the
oracle's result, once waits succeed.

The give-up is made to happen with ``sb_debug_wait_limit(0)``; nothing faults
or hangs (see test_gpu_bounded_wait.py)."""

from __future__ import annotations

import time

import pytest

from stencil_benchmarks_gb300 import _native, serving
from tests.gpu_helpers import bits_equal, mismatch_report
from tests.serving_helpers import download_output, expected_output

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["batched", "plain"])
@pytest.mark.parametrize("other_sync", [False, True])  # another part of the program synchronises meanwhile
def test_requests_run_again(mode, other_sync, lib):
    srv = serving.Server(budget_bytes=1e9, max_batch=4, max_nk=32, slots_per_form=2, keep_outputs=True, mode=mode)
    reqs = [serving.Request(n, op, 60 + n, 40, 24, storage, 100 + n)
            for n, (op, storage) in enumerate([("vadv", "float32"), ("hdiff", "float32"), ("vadv", "float64"),
                                               ("vadv", "bfloat16"), ("hdiff", "float64"), ("vadv", "float32")] * 2)]
    waits = [r for r in reqs if r.op == "vadv" and r.storage != "float64"]
    for r in reqs:
        srv.submit(r)
    errors = 0
    _native.call("sb_debug_wait_limit", 0)
    try:
        for _ in range(200):
            try:
                srv.step()
            except _native.SbError as err:
                assert err.code == _native.SB_ERR_TIMEOUT
                errors += 1
            if other_sync:
                _native.lib().sb_synchronize()
            if errors >= 3:
                break
            time.sleep(0.002)
    finally:
        _native.call("sb_debug_wait_limit", -1)
    assert errors >= 3
    assert not any(r.completed for r in waits)
    deadline = time.monotonic() + 60.0
    while True:
        assert time.monotonic() < deadline
        try:
            if not srv.step():
                break
        except _native.SbError as err:  # launched before the limit was put back
            assert err.code == _native.SB_ERR_TIMEOUT
    assert sorted(r.rid for r in srv.completed) == list(range(len(reqs)))
    for r in reqs:
        got, want = download_output(r), expected_output(r)
        assert bits_equal(got, want), f"{r}: " + mismatch_report(got, want)
        srv.release(r)
    assert srv.pool.in_use == 0
    assert _native.lib().sb_synchronize() == _native.SB_OK
