"""hdiff strips of two columns per lane on rows that no aligned vectors fit, which
AUTO takes for float32, bfloat16 and float-pair arithmetic: strip edges, short
and long row tiles, odd row strides and fields at different offsets, against
the oracle.

float32 arithmetic is the oracle's, operation by operation: no tolerance.
Float pairs: each of hdiff's 11 operations is within 2^-46 of the result's
scale (8 times the largest input), far below the 1e-12 asked for here."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import stencils as ora
from stencil_benchmarks_gb300 import kernels
from stencil_benchmarks_gb300.device import Field
from tests.gpu_helpers import (compute_view, download_like, host_field, interior, round_to_storage, to_device)
from tests.test_gpu_parity import _assert_bits, _run_hdiff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("domain", [(1, 1, 1), (59, 7, 2), (60, 8, 2), (61, 9, 2), (119, 15, 2), (121, 17, 2), (181, 33, 3)])
@pytest.mark.parametrize("halo", [(2, 2, 0), (3, 2, 0), (2, 3, 1)])
@pytest.mark.parametrize("storage", ["float32", "bfloat16"])
def test_strip_edges(storage, domain, halo, lib):
    got, want, _ = _run_hdiff(domain, halo, storage, "float32", seed=sum(domain))
    _assert_bits(got, want, f"strips {storage} {domain} {halo}")


@pytest.mark.parametrize("storage", ["float32", "bfloat16", "float64"])
def test_fields_at_different_offsets(storage, lib):
    """Even row strides, but inp, coeff and out start at different places in a vector."""
    domain, halo = (124, 19, 2), (2, 2, 0)
    compute, oracle = ("float32x2", "float64") if storage == "float64" else ("float32", "float32")
    rng = np.random.Generator(np.random.PCG64(4))
    shape = tuple(d + 2 * h for d, h in zip(domain, halo))
    hosts = {n: host_field(rng.random(shape), storage, halo=halo) for n in ("inp", "coeff", "out")}
    dev = {}
    for shift, (n, h) in enumerate(hosts.items()):
        whole = to_device(h, storage, halo)
        moved = Field.like_host(np.ndarray(shape[:2] + (shape[2] + 1,), h.dtype, strides=h.strides,
                                           buffer=np.zeros(h.nbytes + h.strides[2], np.uint8)), storage, halo)
        dev[n] = Field(moved.buffer, whole.shape, whole.strides, storage, halo, offset=shift * whole.itemsize)
        dev[n].upload(h)
    kernels.hdiff(dev["inp"], dev["coeff"], dev["out"], compute=compute)
    got = interior(download_like(dev["out"], hosts["out"]), domain, halo)
    want = ora.hdiff(compute_view(hosts["inp"], storage, oracle), compute_view(hosts["coeff"], storage, oracle), domain, halo)
    if storage == "float64":
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
    else:
        _assert_bits(got, round_to_storage(want, storage), f"offsets {storage}")


@pytest.mark.parametrize("domain", [(61, 9, 2), (121, 33, 2)])
def test_float_pair(domain, lib):
    halo = (2, 2, 0)
    shape = tuple(d + 2 * h for d, h in zip(domain, halo))
    rng = np.random.Generator(np.random.PCG64(6))
    hosts = {n: host_field(rng.random(shape), halo=halo) for n in ("inp", "coeff", "out")}
    dev = {n: to_device(h, "float64", halo) for n, h in hosts.items()}
    kernels.hdiff(dev["inp"], dev["coeff"], dev["out"], compute="float32x2")
    got = interior(download_like(dev["out"], hosts["out"]), domain, halo)
    want = ora.hdiff(np.array(hosts["inp"]), np.array(hosts["coeff"]), domain, halo)
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
