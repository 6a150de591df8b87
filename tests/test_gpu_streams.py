"""Float32-compute vertical advection of small domains on several streams at
once: launches share the SMs' tensor memory, each with columns for its own
factors only.  Every result is the one of a launch alone."""

from __future__ import annotations

import numpy as np
import pytest

from stencil_benchmarks_gb300 import _native, kernels
from stencil_benchmarks_gb300.device import Field, Stream
from tests.gpu_helpers import VADV_ARGS, VADV_DISTS, bits_equal, download_like, host_field, interior, rng_fields, to_device

pytestmark = pytest.mark.gpu

# factors of 32 to 512 tensor-memory columns a block: levels and warps per block
DOMAINS = [(64, 64, 20), (64, 64, 40), (33, 47, 72), (96, 64, 137), (20, 20, 256), (128, 300, 64), (160, 300, 90), (70, 9, 24)]


@pytest.mark.parametrize("storage", ["float32", "bfloat16"])
def test_side_by_side(storage, lib):
    halo = (1, 1, 0)
    work = []
    for n, domain in enumerate(DOMAINS):
        shape = tuple(d + 2 * h for d, h in zip(domain, halo))
        hosts = [host_field(v, storage, halo=halo) for v in rng_fields(n, shape, VADV_ARGS, VADV_DISTS).values()]
        fields = [to_device(h, storage, halo) for h in hosts]
        out = [Field.like_host(hosts[0], storage, halo) for _ in range(2)]
        kernels.vadv(*fields, (1, 0), out=out[1], compute="float32")
        _native.synchronize()
        work.append((domain, hosts[0], fields, out, Stream()))
    for _ in range(30):
        for _, _, fields, out, stream in work:
            kernels.vadv(*fields, (1, 0), out=out[0], compute="float32", stream=stream)
    _native.synchronize()
    for domain, like, _, out, _ in work:
        got, want = (interior(download_like(o, like), domain, halo) for o in out)
        assert np.any(want) and bits_equal(got, want), domain
