"""Calls of different sizes from several host threads at once: each kernel's
shared-memory limit serves all of them, and every result is the one a call
alone gives."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from stencil_benchmarks_gb300 import _native, kernels
from stencil_benchmarks_gb300.device import Field, Stream
from tests.gpu_helpers import VADV_ARGS, VADV_DISTS, bits_equal, download_like, host_field, interior, rng_fields, to_device

pytestmark = pytest.mark.gpu

CALLS = 400
# shared memory per block from 120 KB to nearly all of it (levels x warps), for each staging form
FORMS = {
    "tma": ("float32", None, [(64, 300, 137), (33, 5, 24), (1, 2, 9), (96, 64, 80)]),
    "rows in tensor memory": ("float32", {"variant": _native.VADV_TMEM, "unroll": 8}, [(96, 64, 20), (33, 9, 256), (64, 30, 130)]),
    "shared memory": ("float32", {"variant": _native.VADV_SMEM}, [(40, 6, 250), (40, 6, 400), (33, 4, 600)]),
}


@pytest.mark.parametrize("name", FORMS)
def test_sizes_side_by_side(name, lib):
    storage, tune, domains = FORMS[name]
    halo = (1, 1, 0)
    errors, work = [], []
    for n, domain in enumerate(domains):
        shape = tuple(d + 2 * h for d, h in zip(domain, halo))
        hosts = [host_field(v, storage, halo=halo) for v in rng_fields(n, shape, VADV_ARGS, VADV_DISTS).values()]
        fields = [to_device(h, storage, halo) for h in hosts]
        out = [Field.like_host(hosts[0], storage, halo) for _ in range(2)]
        work.append((domain, hosts[0], fields, out, Stream()))
    args = _native.tune(**tune) if tune else None
    start = threading.Barrier(len(work))

    def run(fields, out, stream):
        try:
            start.wait()
            for _ in range(CALLS):
                kernels.vadv(*fields, (1, 0), out=out, tune=args, stream=stream)
            stream.synchronize()
        except Exception as err:  # noqa: BLE001 - reported below
            errors.append(err)

    threads = [threading.Thread(target=run, args=(f, out[0], s)) for _, _, f, out, s in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for domain, like, fields, out, _ in work:
        kernels.vadv(*fields, (1, 0), out=out[1], tune=args)
        _native.synchronize()
        got, want = (interior(download_like(o, like), domain, halo) for o in out)
        assert np.any(want) and bits_equal(got, want), domain
