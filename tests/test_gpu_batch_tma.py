"""Batches whose float32 vadv domains are staged by TMA from one queue, whose
hdiff domains are vector strips or (float64) sifted tiles: the per-domain
kernels' results, which the parity tests hold to the oracle, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from stencil_benchmarks_gb300 import _native, kernels
from stencil_benchmarks_gb300.batching import Batch, HdiffDomain, VadvDomain
from stencil_benchmarks_gb300.device import Field
from tests.gpu_helpers import bits_equal, download_like, host_field, interior, mismatch_report, to_device

pytestmark = pytest.mark.gpu


def _domain(op, size, storage, seed, shift=(1, 0), halo_i=None):
    rng = np.random.Generator(np.random.PCG64(seed))
    halo = ((halo_i or 2), 2, 0) if op == "hdiff" else ((halo_i or 1), 1, 0)
    shape = tuple(n + 2 * h for n, h in zip(size, halo))
    names = ("inp", "coeff") if op == "hdiff" else ("stage", "pos", "tens", "tensstage", "wcon")
    span = {"inp": (0, 1), "coeff": (0, 1), "wcon": (-0.5, 0.5)}
    hosts = {n: host_field(rng.uniform(*span.get(n, (-1, 1)), size=shape), storage, halo=halo) for n in names}
    dev = {n: to_device(h, storage, halo) for n, h in hosts.items()}
    like = hosts[names[0]]
    outs = [Field.like_host(like, storage, halo) for _ in range(2)]
    compute = "float64" if storage == "float64" else "float32"
    if op == "hdiff":
        dom = HdiffDomain(dev["inp"], dev["coeff"], outs[0])
        kernels.hdiff(dev["inp"], dev["coeff"], outs[1], compute=compute)
    else:
        fields = [dev[n] for n in names]
        dom = VadvDomain(*fields, out=outs[0], shift=shift)
        kernels.vadv(*fields, shift, out=outs[1], compute=compute)

    def check(what):
        got, want = (interior(download_like(o, like), size, halo) for o in outs)
        assert bits_equal(got, want), f"{what} {op} {size} {storage}: " + mismatch_report(got, want)

    return dom, check


# level strides (halo 1) of 0, 8 and other bytes modulo 16 alone, and together; wcon at i + 1, j + 1 and in place;
# more column groups than warps; level counts around the blocks of 8
SETS = {
    "float32 drift 0": ("float32", [((34, 6, 24), (1, 0)), ((30, 62, 40), (1, 0)), ((62, 30, 17), (1, 0))]),
    "float32 drift 8": ("float32", [((33, 8, 25), (1, 0)), ((64, 5, 32), (0, 1)), ((64, 5, 80), (0, 0))]),
    "float32 mixed": ("float32", [((33, 8, 25), (1, 0)), ((31, 5, 19), (0, 1)), ((34, 6, 64), (0, 0)), ((1, 1, 17), (1, 0))]),
    "float32 many": ("float32", [((510, 126, 18), (1, 0)), ((254, 254, 21), (1, 0)), ((30, 30, 137), (1, 0))]),
    "bfloat16 drift 8": ("bfloat16", [((30, 62, 41), (1, 0)), ((62, 30, 17), (1, 0)), ((126, 94, 66), (1, 0))]),
    "bfloat16 mixed": ("bfloat16", [((33, 5, 30), (0, 1)), ((30, 62, 41), (1, 0)), ((36, 7, 18), (1, 0))]),
    "short columns": ("float32", [((34, 6, 24), (1, 0)), ((34, 6, 5), (1, 0))]),  # not all of them by TMA
}
HDIFF = [(60, 16, 2), (61, 33, 3), (126, 20, 2), (5, 5, 1)]


@pytest.mark.parametrize("name", SETS)
@pytest.mark.parametrize("order", [0, 1])
def test_sets(name, order, lib):
    storage, sizes = SETS[name]
    built = [_domain("vadv", size, storage, 3 + q, shift) for q, (size, shift) in enumerate(sizes)]
    built += [_domain("hdiff", size, storage, 50 + q) for q, size in enumerate(HDIFF)]
    batch = Batch(storage, "float32", max_domains=16, max_nk=137, order=order)
    for _ in range(2):  # the second launch replays the graph
        batch.set([d for d, _ in built])
        batch.launch()
        _native.synchronize()
        for _, check in built:
            check(name)


@pytest.mark.parametrize("storage", ["float64", "float32", "bfloat16"])
@pytest.mark.parametrize("halo_i", [2, 3, 4, 5])
def test_hdiff_rows_at_every_offset(storage, halo_i, lib):
    """Rows that vectors fit, and rows they do not, in one set."""
    built = [_domain("hdiff", size, storage, q, halo_i=halo_i) for q, size in enumerate(HDIFF + [(64, 9, 2), (57, 11, 2)])]
    batch = Batch(storage, max_domains=16, max_nk=8, hdiff_planes=2)
    batch.set([d for d, _ in built])
    batch.launch()
    _native.synchronize()
    for _, check in built:
        check(f"halo {halo_i}")


def test_one_batch_over_sets_of_every_kind(lib):
    """The captured kernels change with the set."""
    batch = Batch("float32", max_domains=8, max_nk=137)
    for name in ("float32 drift 0", "short columns", "float32 drift 8", "float32 mixed", "float32 drift 0"):
        built = [_domain("vadv", size, "float32", 7, shift) for size, shift in SETS[name][1]]
        batch.set([d for d, _ in built])
        batch.launch()
        _native.synchronize()
        for _, check in built:
            check(name)


def test_give_up_is_reported(lib):
    dom, check = _domain("vadv", (64, 20, 24), "float32", 1)
    batch = Batch("float32", max_domains=2, max_nk=32)
    batch.set([dom])
    _native.call("sb_debug_wait_limit", 0)
    try:
        with pytest.raises(_native.SbError) as err:
            batch.launch(timed=True)
        assert err.value.code == _native.SB_ERR_TIMEOUT
        batch.launch()
        assert _native.lib().sb_synchronize() == _native.SB_ERR_TIMEOUT
    finally:
        _native.call("sb_debug_wait_limit", -1)
    batch.launch(timed=True)
    check("after a give-up")
