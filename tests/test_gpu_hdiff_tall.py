"""Domains taller than one kernel's launch grid: AUTO takes the strips whose
blocks cover more rows, as a caller that names them would."""

from __future__ import annotations

import numpy as np
import pytest

from stencil_benchmarks_gb300 import _native, kernels
from tests.gpu_helpers import bits_equal, download_like, host_field, interior, mismatch_report, rng_fields, to_device

pytestmark = pytest.mark.gpu


# rows of 9 elements fit no vectors; tiles of 8 x 2 and 16 rows end at 2^20 rows, JSCAN's at 2^21
@pytest.mark.parametrize("storage,compute", [("float32", "float32"), ("bfloat16", "float32"), ("float64", "float32x2")])
@pytest.mark.parametrize("rows", [(1 << 20) - 16, (1 << 20) + 5])
def test_auto_covers_what_jscan_covers(storage, compute, rows, lib):
    domain, halo = (5, rows, 1), (2, 2, 0)
    shape = tuple(d + 2 * h for d, h in zip(domain, halo))
    hosts = {n: host_field(v, storage, halo=halo) for n, v in rng_fields(2, shape, ("inp", "coeff"), {}).items()}
    dev = {n: to_device(h, storage, halo) for n, h in hosts.items()}
    got = []
    for tune in (None, _native.tune(variant=_native.HDIFF_JSCAN)):
        out = to_device(np.zeros_like(hosts["inp"]), storage, halo)
        kernels.hdiff(dev["inp"], dev["coeff"], out, compute=compute, tune=tune)
        got.append(interior(download_like(out, hosts["inp"]), domain, halo))
    assert np.any(got[0]) and bits_equal(*got), mismatch_report(*got)


def test_a_named_variant_is_refused(lib):
    domain, halo = (60, (1 << 16) + 7, 1), (2, 2, 0)
    shape = tuple(d + 2 * h for d, h in zip(domain, halo))
    host = host_field(np.zeros(shape), "float32", halo=halo)
    inp, coeff, out = (to_device(host, "float32", halo) for _ in range(3))
    with pytest.raises(_native.SbError) as err:
        kernels.hdiff(inp, coeff, out, tune=_native.tune(variant=_native.HDIFF_VSCAN, block_x=64, block_y=1, tile_y=1))
    assert err.value.code == _native.SB_ERR_INVALID
