"""Tiles of the sifted float64 hdiff that are computed in full: every width that
changes the lanes per row (up to 12 and 28 columns), alone and as the last tile
of a row, and heights around the pieces that the warps take, on fields whose
fluxes stay open, are exactly zero, or have zeros beside values.  Bit for bit
against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_hdiff_sift import SIFT, _check

pytestmark = pytest.mark.gpu


def _field(name, shape, rng):
    i, j = np.arange(shape[0])[:, None, None], np.arange(shape[1])[None, :, None]
    if name == "gradient":
        return 100.0 * i + rng.random(shape)
    if name == "constant":
        return np.full(shape, 0.1)
    if name == "linear":
        return 3.0 * i + 2.0 * j + np.zeros(shape)
    if name == "zeros":
        return np.zeros(shape)
    if name == "sparse":
        return np.where(rng.random(shape) < 0.05, rng.uniform(-1, 1, size=shape), 0.0)
    if name == "signed zeros":
        return np.where(rng.random(shape) < 0.5, -0.0, 0.0)
    raise KeyError(name)


@pytest.mark.parametrize("ni", [1, 12, 13, 28, 29, 60, 72, 73, 88, 89])
@pytest.mark.parametrize("nj", [1, 2, 3, 9, 11, 20, 27])
def test_widths_and_heights(ni, nj, lib):
    rng = np.random.Generator(np.random.PCG64(ni + 100 * nj))
    shape = (ni + 4, nj + 4, 2)
    _check(_field("gradient", shape, rng), rng.uniform(-1, 1, size=shape), (ni, nj, 2), (2, 2, 0), f"dense {ni}x{nj}")


@pytest.mark.parametrize("name", ["constant", "linear", "zeros", "sparse", "signed zeros"])
@pytest.mark.parametrize("tune", [SIFT, {"variant": 1}, {"variant": 2}, {"variant": 3}], ids=["sift", "tile", "jscan", "tma"])
@pytest.mark.parametrize("scale", [1.0, 2.0**-1030, 2.0**1010])
def test_zero_fluxes(name, tune, scale, lib):
    """The limiter's rule for products that are a zero or a NaN, in every float64 form."""
    rng = np.random.Generator(np.random.PCG64(3))
    shape = (84, 31, 2)
    _check(_field(name, shape, rng) * scale, rng.uniform(-1, 1, size=shape), (80, 27, 2), (2, 2, 0), f"{name} {scale}", tune)
