"""Performance cases of the stencil backend: what a user has it compute, by
its public Python entry points, over the sizes, element types and options in
use.

Every case is one call of ``stencil_benchmarks_gb300.kernels`` or one launch of
a prepared ``batching.Batch``, on fields that already live on the GPU in the
reference's layout (i unit-stride, then j, then k; halo 2 in i and j for
horizontal diffusion, 1 otherwise) and on the null stream.  Field values have
the distributions of the benchmark workloads: hdiff U[0, 1); vadv
stage/pos/tens/tensstage U[-1, 1), wcon U[-0.5, 0.5); STREAM and the basic
stencils U[0, 1).
"""

from __future__ import annotations

import math

import numpy as np
import torch

from stencil_benchmarks_gb300 import _native, kernels, workloads
from stencil_benchmarks_gb300.array import element_size, layout_strides
from stencil_benchmarks_gb300.batching import Batch, HdiffDomain, VadvDomain
from stencil_benchmarks_gb300.device import Field

DTYPES = {"float64": torch.float64, "float32": torch.float32, "bfloat16": torch.bfloat16}
DTR = 3.0 / 20.0
SHIFTS = ((1, 0), (0, 1), (0, 0))  # wcon columns of the u, v and w components
SCALAR = 3.0
# points of the largest single domain
MAX_POINTS = 512 * 512 * 80


def listed():
    return [
        # The roofline set's domain, a regional weather-model grid, exact float64.
        {"name": "hdiff_f64_512x512x80", "op": "hdiff", "storage": "float64", "compute": "float64",
         "ni": 512, "nj": 512, "nk": 80, "align": 0},
        # The domain of one rank of a decomposed model, also the backend's verification configuration.
        {"name": "hdiff_f64_128x128x64", "op": "hdiff", "storage": "float64", "compute": "float64",
         "ni": 128, "nj": 128, "nk": 64, "align": 0},
        # The roofline domain in single precision, how most operational models run by now.
        {"name": "hdiff_f32_512x512x80", "op": "hdiff", "storage": "float32", "compute": "float32",
         "ni": 512, "nj": 512, "nk": 80, "align": 0},
        # A ragged domain in 16-bit storage with unpadded rows: no row starts on a vector boundary.
        {"name": "hdiff_bf16_391x263x97", "op": "hdiff", "storage": "bfloat16", "compute": "float32",
         "ni": 391, "nj": 263, "nk": 97, "align": 0},
        # The implicit solve of the roofline set, exact float64, with the reference's scratch fields.
        {"name": "vadv_f64_512x512x80", "op": "vadv", "storage": "float64", "compute": "float64",
         "ni": 512, "nj": 512, "nk": 80, "align": 0, "scratch": True},
        # The same solve in single precision.
        {"name": "vadv_f32_512x512x80", "op": "vadv", "storage": "float32", "compute": "float32",
         "ni": 512, "nj": 512, "nk": 80, "align": 0, "scratch": False},
        # The same solve on 16-bit stored fields.
        {"name": "vadv_bf16_512x512x80", "op": "vadv", "storage": "bfloat16", "compute": "float32",
         "ni": 512, "nj": 512, "nk": 80, "align": 0, "scratch": False},
        # The smallest requests of a server, where latency counts and few columns exist.
        {"name": "vadv_f32_96x64x40", "op": "vadv", "storage": "float32", "compute": "float32",
         "ni": 96, "nj": 64, "nk": 40, "align": 0, "scratch": False},
        # A basic stencil of the scaling collection, exact float64.
        {"name": "laplacian_f64_512x512x80", "op": "laplacian", "storage": "float64", "compute": "float64",
         "ni": 512, "nj": 512, "nk": 80, "align": 0, "axes": "xy"},
        # A staggered-grid average on a ragged domain.
        {"name": "average_f32_501x350x60", "op": "average", "storage": "float32", "compute": "float32",
         "ni": 501, "nj": 350, "nk": 60, "align": 0, "axis": 1, "symmetric": True},
        # Many uneven domains in one launch: nested grids, or the queued requests of a server.
        {"name": "batch_f32_64", "op": "batch", "storage": "float32", "domains": 64, "specs": 3},
        # The bandwidth calibration, arrays far beyond L2.
        {"name": "triad_f64_2p27", "op": "triad", "storage": "float64", "n": 1 << 27},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["hdiff", "hdiff", "hdiff", "vadv", "vadv", "vadv", "vadv3", "laplacian", "average", "copy",
                     "batch", "triad"])
    if op == "triad":
        return {"op": op, "storage": rng.choice(["float64", "float32"]), "n": _log_uniform(rng, 1 << 14, 1 << 27)}
    storage = rng.choice(["float64", "float64", "float32", "float32", "bfloat16"])
    if op == "batch":
        most = 6 if storage == "float64" else 48
        return {"op": op, "storage": storage, "domains": rng.randint(2, most), "specs": rng.randint(4, 1 << 20)}
    most = MAX_POINTS // 3 if op == "vadv3" else MAX_POINTS
    while True:
        ni, nj, nk = _log_uniform(rng, 24, 1024), _log_uniform(rng, 24, 1024), rng.randint(8, 137)
        if ni * nj * nk <= most:
            break
    case = {"op": op, "storage": storage, "compute": "float64" if storage == "float64" else "float32",
            "ni": ni, "nj": nj, "nk": nk, "align": rng.choice([0, 0, 128])}
    if op == "hdiff" and storage == "float64":
        case["compute"] = rng.choice(["float64", "float64", "float64", "fixed64"])
    if op in ("vadv", "vadv3"):
        case["scratch"] = storage == "float64" and rng.random() < 0.75
        if case["scratch"]:
            case["compute"] = rng.choice(["float64", "float64", "float64", "float32x2"])
    if op == "laplacian":
        case["axes"] = rng.choice(["xy", "xy", "xyz", "z"])
    if op == "average":
        case["axis"], case["symmetric"] = rng.randint(0, 2), rng.random() < 0.5
    return case


class _Memory:
    """A field's allocation: a torch tensor with the address a Field asks for."""

    def __init__(self, tensor):
        self.tensor = tensor
        self.ptr = tensor.data_ptr()


class _Fields:
    """Fields of one domain, filled from one generator in the order they are asked for."""

    def __init__(self, domain, halo, storage, align, generator):
        self.domain, self.halo, self.storage = domain, halo, storage
        self.generator = generator
        self.shape = tuple(n + 2 * h for n, h in zip(domain, halo))
        size = element_size(storage)
        strides, total = layout_strides(self.shape, size, (2, 1, 0), align)
        self.strides = tuple(s // size for s in strides)
        self.inner = sum(s * h for s, h in zip(self.strides, halo))
        # torch allocations start on 512-byte boundaries: shift the first interior point to an aligned one
        self.offset = (-self.inner) % (align // size) if align else 0
        self.elements = total // size + self.offset

    def field(self, lo=0.0, hi=0.0):
        if hi > lo:
            kind = torch.float64 if self.storage == "float64" else torch.float32
            values = torch.rand(self.elements, dtype=kind, device="cuda", generator=self.generator)
            values = values.mul_(hi - lo).add_(lo).to(DTYPES[self.storage])
        else:
            values = torch.zeros(self.elements, dtype=DTYPES[self.storage], device="cuda")
        return Field(_Memory(values), self.shape, self.strides, self.storage, self.halo,
                     offset=self.offset * element_size(self.storage))


def _view(field, interior=True):
    """The field's interior (or the field with its halo) as a tensor."""
    base = field.buffer.tensor
    start = field.offset // field.itemsize
    shape = field.shape
    if interior:
        start += sum(s * h for s, h in zip(field.strides, field.halo))
        shape = tuple(n - 2 * h for n, h in zip(field.shape, field.halo))
    return base.as_strided(shape, field.strides, start)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)


def _hdiff_fields(make):
    return {"inp": make.field(0.0, 1.0), "coeff": make.field(0.0, 1.0), "out": make.field()}


def _vadv_fields(make):
    fields = {n: make.field(-1.0, 1.0) for n in ("stage", "pos", "tens", "tensstage")}
    return dict(fields, out=make.field())


def _specs(case):
    return workloads.uneven_specs(case["specs"], case["domains"])


def _batch_fields(case, seed):
    generator = _generator(seed)
    found = []
    for spec in _specs(case):
        halo = workloads.HDIFF_HALO if spec.op == "hdiff" else workloads.VADV_HALO
        make = _Fields((spec.ni, spec.nj, spec.nk), halo, case["storage"], 0, generator)
        if spec.op == "hdiff":
            found.append((spec, _hdiff_fields(make)))
        else:
            found.append((spec, dict(_vadv_fields(make), wcon=make.field(-0.5, 0.5))))
    return found


def _inputs(case, seed):
    """The case's fields or arrays, from the seed alone."""
    op = case["op"]
    if op == "batch":
        return _batch_fields(case, seed)
    generator = _generator(seed)
    if op == "triad":
        a = torch.zeros(case["n"], dtype=DTYPES[case["storage"]], device="cuda")
        b, c = (torch.rand(case["n"], dtype=a.dtype, device="cuda", generator=generator) for _ in range(2))
        return {"a": a, "b": b, "c": c}
    halo = workloads.HDIFF_HALO if op == "hdiff" else workloads.VADV_HALO if op.startswith("vadv") else (1, 1, 1)
    make = _Fields((case["ni"], case["nj"], case["nk"]), halo, case["storage"], case["align"], generator)
    if op == "hdiff":
        return _hdiff_fields(make)
    if op in ("vadv", "vadv3"):
        fields = {"components": [_vadv_fields(make) for _ in range(3 if op == "vadv3" else 1)],
                  "wcon": make.field(-0.5, 0.5)}
        if case["scratch"]:
            fields["ccol"], fields["dcol"] = make.field(), make.field()
        return fields
    return {"inp": make.field(0.0, 1.0), "out": make.field()}


def prepare(case, seed):
    state = {"case": case, "in": _inputs(case, seed)}
    if case["op"] == "batch":
        domains = []
        for spec, f in state["in"]:
            if spec.op == "hdiff":
                domains.append(HdiffDomain(f["inp"], f["coeff"], f["out"]))
            else:
                domains.append(VadvDomain(f["stage"], f["pos"], f["tens"], f["tensstage"], f["wcon"], out=f["out"]))
        state["batch"] = Batch(case["storage"], max_domains=case["domains"], max_nk=137)
        state["batch"].set(domains)
    return state


def run(state):
    case, f = state["case"], state["in"]
    op = case["op"]
    if op == "batch":
        state["batch"].launch()
        return [_view(fields["out"]) for _, fields in f]
    if op == "triad":
        kernels.stream_op(_native.STREAM_TRIAD, case["storage"], f["a"].data_ptr(), f["b"].data_ptr(),
                          f["c"].data_ptr(), case["n"], SCALAR)
        return f["a"]
    if op == "hdiff":
        kernels.hdiff(f["inp"], f["coeff"], f["out"], compute=case["compute"])
    elif op == "vadv":
        c = f["components"][0]
        kernels.vadv(c["stage"], c["pos"], c["tens"], c["tensstage"], f["wcon"], SHIFTS[0], ccol=f.get("ccol"),
                     dcol=f.get("dcol"), out=c["out"], compute=case["compute"])
        return _view(c["out"])
    elif op == "vadv3":
        comps = f["components"]
        kernels.vadv3([(c["stage"], c["pos"], c["tens"], c["tensstage"]) for c in comps], f["wcon"],
                      ccol=f.get("ccol"), dcol=f.get("dcol"), outs=[c["out"] for c in comps],
                      compute=case["compute"])
        return [_view(c["out"]) for c in comps]
    elif op == "laplacian":
        kernels.laplacian(f["inp"], f["out"], along=tuple(a in case["axes"] for a in "xyz"), compute=case["compute"])
    elif op == "average":
        kernels.average(f["inp"], f["out"], case["axis"], case["symmetric"], compute=case["compute"])
    else:
        kernels.copy(f["inp"], f["out"])
    return _view(f["out"])


def _work(op, ni, nj, nk, size, case):
    points = ni * nj * nk
    if op == "hdiff":  # inp with its halo, coeff, out; Laplacian 5, two limited fluxes 6, update 5
        return size * ((ni + 4) * (nj + 4) * nk + 2 * points), 16 * points
    if op == "vadv":  # stage, pos, tens, tensstage, out; wcon with one more column
        return size * (5 * points + (ni + 1) * nj * nk), 27 * points
    if op == "vadv3":
        return size * (15 * points + (ni + 1) * (nj + 1) * nk), 81 * points
    if op == "laplacian":
        shape = [n + 2 * (a in case["axes"]) for a, n in zip("xyz", (ni, nj, nk))]
        return size * (math.prod(shape) + points), (3 * len(case["axes"]) - 1) * points
    if op == "average":
        shape = [n + (a == case["axis"]) * (2 if case["symmetric"] else 1) for a, n in enumerate((ni, nj, nk))]
        return size * (math.prod(shape) + points), 2 * points
    return 2 * size * points, 0  # copy


def work(case):
    op, size = case["op"], element_size(case["storage"])
    if op == "triad":
        return {"bytes": 3 * size * case["n"], "flops": 2 * case["n"]}
    if op == "batch":
        parts = [_work(s.op, s.ni, s.nj, s.nk, size, case) for s in _specs(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    found = _work(op, case["ni"], case["nj"], case["nk"], size, case)
    return {"bytes": found[0], "flops": found[1]}


# ---- the same in 64 bits, in plain torch -------------------------------------------------------------------------


def _exact_hdiff(inp, coeff):
    """``inp`` and ``coeff`` with their halo of 2; the interior of the result."""
    lap = 4 * inp[1:-1, 1:-1] - (inp[2:, 1:-1] + inp[:-2, 1:-1] + inp[1:-1, 2:] + inp[1:-1, :-2])
    zero = torch.zeros((), dtype=lap.dtype, device=lap.device)
    x = inp[1:-1, 2:-2]
    flx = lap[1:, 1:-1] - lap[:-1, 1:-1]
    flx = torch.where(flx * (x[1:] - x[:-1]) > 0, zero, flx)
    y = inp[2:-2, 1:-1]
    fly = lap[1:-1, 1:] - lap[1:-1, :-1]
    fly = torch.where(fly * (y[:, 1:] - y[:, :-1]) > 0, zero, fly)
    return inp[2:-2, 2:-2] - coeff[2:-2, 2:-2] * (flx[1:] - flx[:-1] + fly[:, 1:] - fly[:, :-1])


def _exact_vadv(stage, pos, tens, tensstage, wcon, wcon_shifted):
    """Interiors of the fields (the last one shifted); the result's interior."""
    nk = stage.shape[2]

    def level(a, k):
        return a[:, :, k].double()

    def rhs(k):
        return DTR * level(pos, k) + level(tens, k) + level(tensstage, k)

    gcv = 0.25 * (level(wcon_shifted, 1) + level(wcon, 1))
    cs = 0.5 * gcv
    bcol = DTR - cs
    ccol, dcol = [cs / bcol], [(rhs(0) - cs * (level(stage, 1) - level(stage, 0))) / bcol]
    for k in range(1, nk):
        acol = -0.5 * gcv
        below = level(stage, k - 1) - level(stage, k)
        if k < nk - 1:
            gcv = 0.25 * (level(wcon_shifted, k + 1) + level(wcon, k + 1))
            cs = 0.5 * gcv
            bcol = DTR - acol - cs
            right = rhs(k) + (-acol * below - cs * (level(stage, k + 1) - level(stage, k)))
            divided = 1.0 / (bcol - ccol[-1] * acol)
            ccol.append(cs * divided)
            dcol.append((right - dcol[-1] * acol) * divided)
        else:
            right = rhs(k) + -acol * below
            dcol.append((right - dcol[-1] * acol) / (DTR - acol - ccol[-1] * acol))
    data = dcol[-1]
    out = torch.empty(stage.shape, dtype=torch.float64, device=stage.device)
    out[:, :, nk - 1] = DTR * (data - level(pos, nk - 1))
    for k in range(nk - 2, -1, -1):
        data = dcol[k] - ccol[k] * data
        out[:, :, k] = DTR * (data - level(pos, k))
    return out


def _shifted(field, shift):
    whole = _view(field, interior=False)
    return whole[tuple(slice(h + s, h + s + n - 2 * h) for n, h, s in zip(field.shape, field.halo, shift))]


def _exact_component(c, wcon, shift):
    return _exact_vadv(*(_view(c[n]) for n in ("stage", "pos", "tens", "tensstage")), _view(wcon),
                       _shifted(wcon, shift + (0,)))


def exact(case, seed):
    op, f = case["op"], _inputs(case, seed)
    if op == "triad":
        return f["b"].double() + SCALAR * f["c"].double()
    if op == "batch":
        return [_exact_hdiff(_view(d["inp"], False).double(), _view(d["coeff"], False).double())
                if spec.op == "hdiff" else _exact_component(d, d["wcon"], SHIFTS[0]) for spec, d in f]
    if op == "hdiff":
        return _exact_hdiff(_view(f["inp"], False).double(), _view(f["coeff"], False).double())
    if op == "vadv":
        return _exact_component(f["components"][0], f["wcon"], SHIFTS[0])
    if op == "vadv3":
        return [_exact_component(c, f["wcon"], s) for c, s in zip(f["components"], SHIFTS)]

    def at(shift):
        return _shifted(f["inp"], tuple(shift)).double()

    if op == "laplacian":
        result = torch.zeros((case["ni"], case["nj"], case["nk"]), dtype=torch.float64, device="cuda")
        for axis in (a for a in range(3) if "xyz"[a] in case["axes"]):
            step = np.eye(3, dtype=int)[axis]
            result += 2 * at((0, 0, 0)) - at(step) - at(-step)
        return result
    if op == "average":
        step = np.eye(3, dtype=int)[case["axis"]]
        return 0.5 * (at(step) + at(-step if case["symmetric"] else 0 * step))
    return at((0, 0, 0))
