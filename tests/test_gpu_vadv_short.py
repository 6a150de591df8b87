"""Float32-compute vertical advection around the level counts and sizes where
AUTO changes between shared-memory and TMA-staged columns, and the TMA-staged
form itself on short columns: bit for bit against the oracle."""

from __future__ import annotations

import pytest

from stencil_benchmarks_gb300 import _native
from tests.test_gpu_parity import _assert_bits, _run_vadv
from tests.test_gpu_vadv_tma import CASES, domain_with

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,drift", CASES)
@pytest.mark.parametrize("nk", [9, 16, 17, 18])
def test_tma_form(storage, drift, nk, lib):
    domain = domain_with(drift, 4 if storage == "float32" else 2, nk)
    got, want = _run_vadv(domain, (1, 1, 0), storage, "float32", seed=nk, tune=_native.tune(variant=_native.VADV_TMEM))
    _assert_bits(got, want, f"vadv tma {storage} {domain}")


@pytest.mark.parametrize("storage", ["float32", "bfloat16"])
@pytest.mark.parametrize("nk", [2, 8, 9, 19, 20])
@pytest.mark.parametrize("nj", [5, 1023, 1024])  # two column groups each: 2046 and 2048 of them
def test_auto(storage, nk, nj, lib):
    got, want = _run_vadv((34, nj, nk), (1, 1, 0), storage, "float32", seed=nk)
    _assert_bits(got, want, f"vadv auto {storage} {nk} {nj}")


@pytest.mark.parametrize("nk", [12, 19, 20])
def test_auto_with_scratch(nk, lib):
    got, want = _run_vadv((70, 9, nk), (1, 1, 0), "float32", "float32", seed=nk, use_scratch=True)
    _assert_bits(got, want, f"vadv auto with scratch {nk}")
