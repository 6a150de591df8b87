"""The three components of vertical advection where a result overwrites a field
that another component reads: as three calls in turn, u before v before w."""

from __future__ import annotations

import numpy as np
import pytest

from stencil_benchmarks_gb300 import _native, kernels
from stencil_benchmarks_gb300.device import Field
from tests.gpu_helpers import VADV_ARGS, VADV_DISTS, bits_equal, download_like, host_field, interior, rng_fields, to_device

pytestmark = pytest.mark.gpu

SHIFTS = ((1, 0), (0, 1), (0, 0))


# which field the last component's result overwrites: wcon, which u and v read at i + 1 and j + 1, or a field of u
@pytest.mark.parametrize("target", ["wcon", "stage", "tensstage"])
@pytest.mark.parametrize("storage,domain", [("float32", (70, 33, 24)), ("bfloat16", (46, 20, 40)), ("float64", (40, 9, 12))])
def test_last_result(storage, domain, target, lib):
    halo = (1, 1, 0)
    shape = tuple(d + 2 * h for d, h in zip(domain, halo))
    got = []
    for fused in (True, False):
        comps = []
        for c in range(3):
            vals = rng_fields(c, shape, VADV_ARGS, VADV_DISTS)
            hosts = [host_field(v, storage, halo=halo) for v in vals.values()]
            comps.append([to_device(h, storage, halo) for h in hosts])
        wcon = comps[0][4]
        like = hosts[0]
        outs = [Field.like_host(like, storage, halo) for _ in range(2)]
        outs.append({"wcon": wcon, "stage": comps[0][0], "tensstage": comps[0][3]}[target])
        if fused:
            kernels.vadv3([tuple(c[:4]) for c in comps], wcon, outs=outs)
        else:
            for c, out, shift in zip(comps, outs, SHIFTS):
                kernels.vadv(*c[:4], wcon, shift, out=out)
        _native.synchronize()
        got.append([interior(download_like(o, like), domain, halo) for o in outs])
    for name, g, w in zip("uvw", *got):
        assert np.any(g) and bits_equal(g, w), f"{target} {name}"
