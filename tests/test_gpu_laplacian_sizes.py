"""The float64 Laplacian strips of domains large enough for the split between
fp64 and integer arithmetic (the smaller ones of test_gpu_laplacian_split.py
run all fp64): the same axis sets and special values, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import stencils as ora
from stencil_benchmarks_gb300 import kernels
from tests.gpu_helpers import (compute_view, download_like, host_field, interior, rng_fields, round_to_storage, to_device)
from tests.test_gpu_parity import _assert_bits

pytestmark = pytest.mark.gpu


# 10 warps per SM and more on any GPU of up to 160 SMs; partial strips and an odd plane
@pytest.mark.parametrize("domain", [(33, 131, 97), (100, 9, 301)])
@pytest.mark.parametrize("along", [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1)])
@pytest.mark.parametrize("storage", ["float64", "float32"])
def test_split(storage, along, domain, lib):
    halo, along = (1, 1, 1), tuple(map(bool, along))
    shape = tuple(d + 2 for d in domain)
    vals = rng_fields(sum(domain), shape, ("inp", "out"), {})
    rng = np.random.Generator(np.random.PCG64(7))
    pick = rng.random(size=shape)
    vals["inp"][pick < 0.3] = 0.0
    vals["inp"][rng.random(size=shape) < 0.4] *= -1.0
    for lo, value in ((0.90, 1e-40 if storage == "float32" else 3e-310), (0.92, 3e38 if storage == "float32" else 1.5e308),
                      (0.94, np.inf), (0.95, np.nan), (0.96, 0.25)):
        vals["inp"][pick > lo] = value
    hosts = {n: host_field(v, storage, halo=halo) for n, v in vals.items()}
    dev = {n: to_device(h, storage, halo) for n, h in hosts.items()}
    kernels.laplacian(dev["inp"], dev["out"], along, compute="float64")
    got = interior(download_like(dev["out"], hosts["out"]), domain, halo)
    with np.errstate(all="ignore"):
        want = round_to_storage(ora.laplacian(compute_view(hosts["inp"], storage, "float64"), domain, halo, along), storage)
    _assert_bits(got, want, f"laplacian {along} {storage} {domain}")
