"""Which launch shapes the batch autotuner times, and which cached results it
trusts (CPU: the batch and the device are stand-ins)."""

from __future__ import annotations

import json
from types import SimpleNamespace

import pytest

from stencil_benchmarks_gb300 import _native, autotune
from stencil_benchmarks_gb300.batching import HdiffDomain, VadvDomain


def _field(nk):
    return SimpleNamespace(shape=(12, 12, nk), halo=(2, 2, 0))


def _domains(nk=40):
    f = _field(nk)
    return [HdiffDomain(f, f, f), VadvDomain(f, f, f, f, f)]


FORMS = [("float64", "float64"), ("float32", "float32"), ("bfloat16", "float32"), ("float64", "float32x2")]


@pytest.mark.parametrize("storage,compute", FORMS)
def test_the_librarys_choice_comes_first(storage, compute):
    found = autotune.candidates_for(storage, compute, _domains())
    assert found[0] == {} and all(p in autotune.DEFAULT_CANDIDATES for p in found[1:])


def test_what_a_form_ignores_is_not_timed_twice():
    def differing(found, *ignored):
        rest = [tuple(sorted((k, v) for k, v in p.items() if k not in ignored)) for p in found[1:]]
        return len(rest) == len(set(rest))

    assert differing(autotune.candidates_for("float64", "float64", _domains()), "block", "hdiff_rows")
    tensor = [p for p in autotune.candidates_for("float32", "float32", _domains())[1:] if p["vadv_block"] == 32]
    assert differing([{}] + tensor, "vadv_blocks_per_sm", "order")
    # the order counts where short columns may run as bucket kernels, the blocks per SM above 256 levels
    short = [p for p in autotune.candidates_for("float32", "float32", _domains(12))[1:] if p["vadv_block"] == 32]
    assert not differing([{}] + short, "order")
    tall = [p for p in autotune.candidates_for("float32", "float32", _domains(300))[1:] if p["vadv_block"] == 32]
    assert not differing([{}] + tall, "vadv_blocks_per_sm")
    # every candidate of a form that ignores nothing
    assert len(autotune.candidates_for("float64", "float32x2", _domains())) == 1 + len(autotune.DEFAULT_CANDIDATES)


class _Batch:
    timed = 0

    def __init__(self, *args, **kw):
        pass

    def set(self, domains):
        pass

    def launch(self, stream=None, timed=False):
        _Batch.timed += 1
        return 1.0

    def close(self):
        pass


def test_results_of_another_revision_are_timed_again(tmp_path, monkeypatch):
    monkeypatch.setenv("SBGB300_TUNE_CACHE", str(tmp_path / "cache.json"))
    monkeypatch.setattr(autotune, "Batch", _Batch)
    monkeypatch.setattr(_native, "current_device", lambda: 0)
    monkeypatch.setattr(_native, "device_info", lambda d: {"name": "gpu"})
    revision = 7
    monkeypatch.setattr(_native, "lib", lambda: SimpleNamespace(sb_version=lambda: revision))
    doms = _domains()
    # as written before the key named a revision
    (tmp_path / "cache.json").write_text(json.dumps(
        {"|".join(["gpu", "float32", "float32", autotune.signature(doms)]): {"params": {"vadv_block": 64}, "seconds": 0.5}}))
    best, results = autotune.autotune_batch("float32", doms, 40)
    assert best == {} and results and _Batch.timed
    assert autotune.autotune_batch("float32", doms, 40) == ({}, [])  # cached now
    revision = 8
    assert autotune.autotune_batch("float32", doms, 40)[1]  # the kernels have changed
