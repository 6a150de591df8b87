"""TMA-staged float32 vertical advection (csrc/vadv_tma.cuh), which AUTO picks
for float32 compute: bit-identical to the oracle at the edges of its 8-level
stages, of the 32-column groups and of the ring that runs on across column
groups, for every level stride modulo the 16 bytes of a tensor stride, and a
give-up of its bounded waits is reported.

No tolerance: the arithmetic is the oracle's, operation by operation."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle import stencils as ora
from stencil_benchmarks_gb300 import _native, kernels
from tests.gpu_helpers import (VADV_ARGS, VADV_DISTS, compute_view, download_like, host_field, interior, rng_fields,
                               round_to_storage, to_device)
from tests.test_gpu_parity import _assert_bits, _run_vadv, _run_vadv3

pytestmark = pytest.mark.gpu


def domain_with(drift, size, nk):
    """A domain of more than one column group whose level stride (halo 1) is ``drift`` modulo 16 bytes."""
    for ni in range(33, 80):
        for nj in (5, 6):
            if (ni + 2) * (nj + 2) * size % 16 == drift:
                return ni, nj, nk
    raise AssertionError(drift)


CASES = [("float32", d) for d in (0, 4, 8, 12)] + [("bfloat16", d) for d in (0, 2, 4, 6, 8, 10, 12, 14)]


@pytest.mark.parametrize("storage,drift", CASES)
@pytest.mark.parametrize("nk", [9, 16, 17, 18, 25, 80, 129, 256])
def test_levels_and_strides(storage, drift, nk, lib):
    domain = domain_with(drift, 4 if storage == "float32" else 2, nk)
    got, want = _run_vadv(domain, (1, 1, 0), storage, "float32", seed=nk + drift)
    _assert_bits(got, want, f"vadv tma {storage} {domain}")


@pytest.mark.parametrize("shift", [(1, 0), (0, 1), (0, 0)])
@pytest.mark.parametrize("storage,domain,halo", [("float32", (33, 9, 14), (1, 1, 1)), ("float32", (1, 7, 21), (3, 2, 1)),
                                                 ("float32", (66, 3, 31), (2, 1, 0)), ("bfloat16", (97, 4, 15), (3, 2, 0)),
                                                 ("bfloat16", (40, 6, 19), (1, 1, 2))])
def test_shifts_and_offsets(storage, domain, halo, shift, lib):
    got, want = _run_vadv(domain, halo, storage, "float32", seed=3, shift=shift)
    _assert_bits(got, want, f"vadv tma {storage} {domain} {halo} {shift}")


@pytest.mark.parametrize("storage,domain", [("float32", (70, 1400, 14)), ("bfloat16", (33, 1001, 16)),
                                            ("float32", (32, 153, 9))])
def test_rings_run_on_across_groups(storage, domain, lib):
    """More column groups than warps: the ring is refilled with the next group's levels."""
    got, want = _run_vadv(domain, (1, 1, 0), storage, "float32", seed=5)
    _assert_bits(got, want, f"vadv tma {storage} {domain}")


@pytest.mark.parametrize("storage,domain", [("float32", (70, 33, 17)), ("float32", (33, 1000, 9)),
                                            ("bfloat16", (46, 20, 22))])
def test_three_components(storage, domain, lib):
    got, want = _run_vadv3(domain, (1, 1, 1), storage, "float32", seed=7)
    for c, g, w in zip("uvw", got, want):
        _assert_bits(g, w, f"vadv3 tma {c} {storage} {domain}")


def test_reciprocal_is_exact_over_its_range(lib):
    """Every float32 with 2^-125 <= |d| <= 2^125, against the correctly rounded reciprocal."""
    checked, wrong = ctypes.c_int64(), ctypes.c_int64()
    _native.call("sb_debug_rcp_f32", ctypes.byref(checked), ctypes.byref(wrong))
    assert checked.value == 2 * (250 * 2**23 + 1) and wrong.value == 0


@pytest.mark.parametrize("storage", ["float32", "bfloat16"])
@pytest.mark.parametrize("scale", [2.0**-127, 2.0**126, 0.0])
def test_pivots_outside_the_reciprocals_range(storage, scale, lib):
    """Blocks of levels are computed once more with the general reciprocal: columns whose wcon makes
    the pivot tiny, huge or exactly dtr / 0 somewhere, beside ordinary ones."""
    domain, halo = (40, 5, 30), (1, 1, 0)
    shape = tuple(d + 2 * h for d, h in zip(domain, halo))
    vals = rng_fields(9, shape, VADV_ARGS, VADV_DISTS)
    rng = np.random.Generator(np.random.PCG64(10))
    # (dtr + cs(k-1)) - cs(k) is scale where wcon jumps by 8 * dtr, or huge where wcon is
    wcon = np.full(shape, 0.0)
    wcon[:, :, 12:] = np.float32(0.6) if scale < 1 else 4 * scale
    wcon = np.where(rng.random(shape[:2] + (1,)) < 0.5, wcon * (1 + scale if scale < 1 else 1), vals["wcon"])
    vals["wcon"] = wcon
    with np.errstate(over="ignore"):  # to infinity in the storage type, as intended
        hosts = {n: host_field(v, storage, halo=halo) for n, v in vals.items()}
    dev = {n: to_device(h, storage, halo) for n, h in hosts.items()}
    kernels.vadv(*(dev[n] for n in VADV_ARGS), (1, 0), compute="float32")
    got = interior(download_like(dev["utensstage"], hosts["utensstage"]), domain, halo)
    with np.errstate(all="ignore"):
        want = ora._vadv_component(*(compute_view(hosts[n], storage, "float32") for n in VADV_ARGS), domain, halo, 1, 0)
        want = round_to_storage(want, storage)
    if storage == "bfloat16":  # NaN bit patterns differ: compare as values
        got, want = (ora.bf16_bits_to_f32(np.ascontiguousarray(a)).reshape(a.shape) for a in (got, want))
    _assert_bits(got, want, f"vadv tma pivots {storage} {scale}")


def test_give_up_is_reported(lib):
    domain, halo = (64, 6, 20), (1, 1, 0)
    shape = tuple(d + 2 * h for d, h in zip(domain, halo))
    fields = [to_device(host_field(v, "float32", halo=halo), "float32", halo)
              for v in rng_fields(1, shape, VADV_ARGS, VADV_DISTS).values()]
    args = [ctypes.c_void_p(f.interior_ptr) for f in fields] + [ctypes.c_void_p(fields[3].interior_ptr), None, None]
    t = ctypes.c_double(0.0)

    def launch(time):
        return _native.lib().sb_vadv(_native.SB_F32, _native.SB_F32, *args, *domain, *fields[0].strides, 1, 0, None,
                                     None, time)

    _native.call("sb_debug_wait_limit", 0)
    try:
        assert launch(ctypes.byref(t)) == _native.SB_ERR_TIMEOUT  # by the timed call itself
        assert launch(None) == _native.SB_OK
        assert _native.lib().sb_synchronize() == _native.SB_ERR_TIMEOUT
    finally:
        _native.call("sb_debug_wait_limit", -1)
    assert launch(ctypes.byref(t)) == _native.SB_OK
