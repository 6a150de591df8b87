"""Exact float64 hdiff that evaluates only the fluxes the limiter may let through
(csrc/hdiff_sift.cuh), AUTO's choice for float64: bit-identical to the oracle
where fluxes are closed, open or undecided, on full and cut tiles, and on the
values that make a tile be computed in full.

No tolerance: the result is defined bit by bit."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import stencils as ora
from stencil_benchmarks_gb300 import _native, kernels
from tests.gpu_helpers import download_like, host_field, interior, to_device
from tests.test_gpu_parity import _assert_bits, _run_hdiff

pytestmark = pytest.mark.gpu

SIFT = {"variant": _native.HDIFF_SIFT}


def _check(inp, coeff, domain, halo, what, tune=SIFT):
    hosts = {"inp": host_field(inp, halo=halo), "coeff": host_field(coeff, halo=halo),
             "out": host_field(np.full(inp.shape, 7.0), halo=halo)}
    dev = {n: to_device(h, "float64", halo) for n, h in hosts.items()}
    kernels.hdiff(dev["inp"], dev["coeff"], dev["out"], tune=_native.tune(**tune) if tune else None)
    whole = download_like(dev["out"], hosts["out"])
    got = interior(whole, domain, halo)
    with np.errstate(all="ignore"):
        want = ora.hdiff(np.array(hosts["inp"]), np.array(hosts["coeff"]), domain, halo)
    _assert_bits(got, want, what)
    outside = np.ones(inp.shape, dtype=bool)
    outside[ora.inner_slice(domain, halo)] = False
    assert np.all(whole[outside] == 7.0), f"{what}: wrote outside the interior"


# one column, row and plane; a tile less, exactly and plus one; cut tiles in both directions
@pytest.mark.parametrize("domain", [(1, 1, 1), (59, 19, 2), (60, 20, 2), (61, 21, 2), (61, 17, 2), (121, 41, 3), (128, 128, 4), (7, 50, 2)])
@pytest.mark.parametrize("halo", [(2, 2, 0), (3, 2, 1)])
def test_tiles(domain, halo, lib):
    got, want, _ = _run_hdiff(domain, halo, tune=_native.tune(**SIFT), seed=sum(domain))
    _assert_bits(got, want, f"sift {domain} {halo}")


@pytest.mark.parametrize("layout,alignment", [((0, 1, 2), 0), ((1, 2, 0), 64), ((2, 1, 0), 128)])
def test_layouts(layout, alignment, lib):
    got, want, _ = _run_hdiff((70, 35, 5), (2, 2, 0), layout=layout, alignment=alignment, tune=_native.tune(**SIFT))
    _assert_bits(got, want, f"sift layout {layout}")


def _fields(name, shape, rng):
    i, j, k = np.meshgrid(*(np.arange(n, dtype=np.float64) for n in shape), indexing="ij")
    if name == "uniform":
        return rng.random(shape)
    if name == "signed":
        return rng.uniform(-1, 1, size=shape)
    if name == "smooth":  # nearly every flux is closed
        return 280.0 + 10 * np.sin(0.05 * i) * np.cos(0.07 * j) + 0.1 * k
    if name == "very smooth":  # third differences below the fixed-point unit: undecided
        return 280.0 + 1e-7 * np.sin(0.05 * i + 0.03 * j)
    if name == "gradient":  # half the fluxes pass: tiles computed in full
        return 100.0 * i + rng.random(shape)
    if name == "patchy":  # both kinds of tile
        return np.where(i < 61, rng.random(shape), 100.0 * j + rng.random(shape))
    if name == "constant":
        return np.full(shape, 0.1)
    if name == "coarse":  # exact ties and equal neighbours
        return rng.integers(0, 4, size=shape) / 4.0
    if name == "wide":  # magnitudes over 60 binades
        return rng.uniform(-1, 1, size=shape) * 2.0 ** rng.integers(-60, 1, size=shape)
    if name == "zeros":
        return np.where(rng.random(shape) < 0.5, 0.0, rng.random(shape))
    raise KeyError(name)


NAMES = ["uniform", "signed", "smooth", "very smooth", "gradient", "patchy", "constant", "coarse", "wide", "zeros"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("scale", [1.0, 2.0**-470, 2.0**-473, 2.0**-1030, 2.0**1000])
def test_fields(name, scale, lib):
    domain, halo = (125, 37, 2), (2, 2, 0)
    rng = np.random.Generator(np.random.PCG64(17))
    shape = tuple(d + 2 * h for d, h in zip(domain, halo))
    _check(_fields(name, shape, rng) * scale, rng.uniform(-1, 1, size=shape), domain, halo, f"sift {name} {scale}")


@pytest.mark.parametrize("where", ["inp", "coeff"])
@pytest.mark.parametrize("value", [-0.0, np.inf, np.nan, 1.7e308, 5e-324, -1e-310])
def test_special_values(where, value, lib):
    """A few special values among ordinary ones; other tiles keep to the sifted path."""
    domain, halo = (130, 40, 3), (2, 2, 0)
    rng = np.random.Generator(np.random.PCG64(5))
    shape = tuple(d + 2 * h for d, h in zip(domain, halo))
    fields = {"inp": rng.uniform(-1, 1, size=shape), "coeff": rng.uniform(-1, 1, size=shape)}
    fields[where][rng.random(shape) < 0.001] = value
    _check(fields["inp"], fields["coeff"], domain, halo, f"sift {where} {value}")


def test_auto_takes_it(lib):
    rng = np.random.Generator(np.random.PCG64(8))
    shape = (104, 44, 3)
    _check(rng.random(shape), rng.random(shape), (100, 40, 3), (2, 2, 0), "auto", tune=None)
    with pytest.raises(_native.SbError) as err:
        _run_hdiff((40, 20, 2), (2, 2, 0), "float32", "float32", tune=_native.tune(**SIFT))
    assert err.value.code == _native.SB_ERR_UNSUPPORTED
