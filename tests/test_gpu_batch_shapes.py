"""Batches whose launch shape follows the installed set: capacities far above
the set's columns, columns of 9 to 16 levels, items of several column groups,
sets that change the shape of a captured graph.  The per-domain kernels'
results, bit for bit."""

from __future__ import annotations

import pytest

from stencil_benchmarks_gb300 import _native
from stencil_benchmarks_gb300.batching import Batch
from tests.test_gpu_batch_tma import _domain

pytestmark = pytest.mark.gpu

U, V, W = (1, 0), (0, 1), (0, 0)


def _run(batch, built, what):
    batch.set([d for d, _ in built])
    for _ in range(2):  # the second launch replays the graph
        batch.launch()
    _native.synchronize()
    for _, check in built:
        check(what)


@pytest.mark.parametrize("storage", ["float32", "bfloat16"])
@pytest.mark.parametrize("max_nk", [80, 256, 257, 600])
def test_capacities(storage, max_nk, lib):
    sizes = [((34, 6, 24), U), ((62, 30, 9), U), ((64, 5, 80), V), ((33, 8, 16), W), ((1, 1, 17), U)]
    built = [_domain("vadv", size, storage, q, shift) for q, (size, shift) in enumerate(sizes)]
    _run(Batch(storage, max_domains=8, max_nk=max_nk), built, f"capacity {max_nk}")


# short columns beside hdiff: items of 2 and 3 groups with a remainder, of tall columns one; alone: the bucket
# kernels, and (bfloat16, 20 levels) items of two groups again
SETS = {
    "beside hdiff": [("vadv", (33, 5000, 12), U), ("vadv", (65, 2501, 9), U), ("vadv", (40, 7, 60), V), ("hdiff", (61, 33, 2), U)],
    "two groups": [("vadv", (33, 5001, 16), W), ("vadv", (30, 9, 33), U), ("hdiff", (61, 33, 2), U)],
    "alone": [("vadv", (33, 5000, 12), U), ("vadv", (65, 2501, 9), U)],
    "many": [("vadv", (33, 10003, 20), U), ("vadv", (31, 50, 19), U)],
    "few": [("vadv", (64, 48, 12), U), ("vadv", (64, 48, 9), W)],
}


@pytest.mark.parametrize("storage", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", SETS)
def test_short_columns(storage, name, lib):
    built = [_domain(op, size, storage, q, shift) for q, (op, size, shift) in enumerate(SETS[name])]
    _run(Batch(storage, max_domains=8, max_nk=64), built, name)


def test_a_captured_graph_follows_the_set(lib):
    batch = Batch("float32", max_domains=8, max_nk=256)
    for sizes in ([(34, 6, 256)], [(34, 6, 9), (62, 30, 12)], [(34, 6, 80), (33, 8, 17)], [(33, 12000, 10), (30, 9, 64)],
                  [(34, 6, 256), (34, 6, 9)], [(34, 6, 5)], [(34, 6, 256)]):
        _run(batch, [_domain("vadv", size, "float32", 7) for size in sizes], f"set {sizes}")


def test_info_reports_the_block_that_runs(lib):
    assert Batch("float64", block=256).info()["block"] == 128  # exact float64 has one block size
    assert Batch("float32", block=256).info()["block"] == 256
