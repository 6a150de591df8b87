"""Horizontal diffusion whose result overwrites the coefficients (out is the
coeff field): every coefficient is read before its point is written, in every
form, alone and in a batch.  Bit for bit against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import stencils as ora
from stencil_benchmarks_gb300 import _native, kernels
from stencil_benchmarks_gb300.batching import Batch, HdiffDomain
from tests.gpu_helpers import (bits_equal, compute_view, download_like, host_field, interior, mismatch_report,
                               rng_fields, round_to_storage, to_device)

pytestmark = pytest.mark.gpu

HALO = (2, 2, 0)
FORMS = [("float64", "float64"), ("float32", "float32"), ("bfloat16", "float32"), ("float32", "float64")]


def _case(domain, storage, compute, seed):
    shape = tuple(d + 2 * h for d, h in zip(domain, HALO))
    hosts = {n: host_field(v, storage, halo=HALO) for n, v in rng_fields(seed, shape, ("inp", "coeff"), {}).items()}
    dev = {n: to_device(h, storage, HALO) for n, h in hosts.items()}

    def check(what):
        got = interior(download_like(dev["coeff"], hosts["coeff"]), domain, HALO)
        want = round_to_storage(ora.hdiff(compute_view(hosts["inp"], storage, compute),
                                          compute_view(hosts["coeff"], storage, compute), domain, HALO), storage)
        assert bits_equal(got, want), f"{what} {domain} {storage}: " + mismatch_report(got, want)

    return dev["inp"], dev["coeff"], check


@pytest.mark.parametrize("storage,compute", FORMS)
@pytest.mark.parametrize("domain", [(128, 40, 3), (61, 21, 2), (5, 3, 1)])
def test_auto(storage, compute, domain, lib):
    inp, coeff, check = _case(domain, storage, compute, 3)
    kernels.hdiff(inp, coeff, coeff, compute=compute)
    check("auto")


def test_sift(lib):
    inp, coeff, check = _case((125, 47, 2), "float64", "float64", 4)
    kernels.hdiff(inp, coeff, coeff, tune=_native.tune(variant=_native.HDIFF_SIFT))
    check("sift")


@pytest.mark.parametrize("storage", ["float64", "float32", "bfloat16"])
def test_batch(storage, lib):
    """Beside domains with a result field of their own."""
    compute = "float64" if storage == "float64" else "float32"
    built = [_case(d, storage, compute, q) for q, d in enumerate([(70, 33, 3), (124, 20, 2), (9, 50, 2)])]
    inp, coeff, _ = _case((64, 30, 2), storage, compute, 9)
    own = to_device(np.zeros_like(host_field(np.zeros((68, 34, 2)), storage, halo=HALO)), storage, HALO)
    batch = Batch(storage, max_domains=8, max_nk=8)
    batch.set([HdiffDomain(i, c, c) for i, c, _ in built] + [HdiffDomain(inp, coeff, own)])
    batch.launch()
    _native.synchronize()
    for _, _, check in built:
        check("batch")
