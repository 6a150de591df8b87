"""Vector strips of every tile height that the dispatch picks by the domain's
size, and the hand-over to JSCAN: the bits of explicit JSCAN strips, which the
parity tests hold to the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from stencil_benchmarks_gb300 import _native, kernels
from tests.gpu_helpers import bits_equal, download_like, host_field, interior, mismatch_report, rng_fields, to_device

pytestmark = pytest.mark.gpu

CASES = [
    ("float32", "float32", (261, 130, 300)),  # odd rows, tiles of 16 rows
    ("float32", "float32", (131, 50, 9)),  # of 8
    ("float64", "float32x2", (124, 50, 9)),  # aligned, of 8
    ("float64", "float32x2", (1004, 61, 240)),  # aligned, of 16
    ("float64", "float32x2", (1001, 61, 240)),  # odd rows, of 16
    ("float64", "float32x2", (61, 121, 480)),  # JSCAN leaves fewer lanes idle
]


@pytest.mark.parametrize("storage,compute,domain", CASES)
def test_same_bits_as_jscan(storage, compute, domain, lib):
    halo = (2, 2, 0)
    shape = tuple(d + 2 * h for d, h in zip(domain, halo))
    hosts = {n: host_field(v, storage, halo=halo) for n, v in rng_fields(5, shape, ("inp", "coeff"), {}).items()}
    dev = {n: to_device(h, storage, halo) for n, h in hosts.items()}
    got = []
    for tune in (None, _native.tune(variant=_native.HDIFF_JSCAN)):
        out = to_device(np.zeros_like(hosts["inp"]), storage, halo)
        kernels.hdiff(dev["inp"], dev["coeff"], out, compute=compute, tune=tune)
        got.append(interior(download_like(out, hosts["inp"]), domain, halo))
    assert np.any(got[0]) and bits_equal(*got), mismatch_report(*got)
