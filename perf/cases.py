"""Timed cases of the transfer path: what a program that uses this package has it do, through the
public entry points, from a few probe points to 3.2e7 particles.

Kinds of case
  gather      interpolate!(out, field, points, scheme, traversal) on the reference's layouts
  scatter     anterpolate!(field, points, quantities, scheme[, alpha, beta]) on the same layouts
  order       point_traversal_order!(...) for points that have moved, then the gather in that order
  step        the resident form's particle step: bins rebuilt, gather, scatter, the deposit read back
  track       a new field loaded, points displaced, wrapped and re-binned in one call, then gathered
  batch       many instances of uneven sizes: batched bins builds and one batch, a captured CUDA graph
  served      requests of mixed sizes to the request loop, waited for together
  nufft2      interpolate! of a field in spectral representation with a NUFFT plan
  nufft1      anterpolate! into a field in spectral representation with a NUFFT plan

A case's sizes are in the case; everything else comes from the seed.
"""
from __future__ import annotations

import importlib.util
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

TWO_PI = 2 * math.pi


def _package():
    """The package, whose directory's name holds a dot, as the module gbgperiodicfields_gb300."""
    name = "gbgperiodicfields_gb300"
    if name not in sys.modules:
        directory = Path(__file__).resolve().parent.parent / "gbgperiodicfields.jl_gb300"
        spec = importlib.util.spec_from_file_location(name, directory / "__init__.py",
                                                      submodule_search_locations=[str(directory)])
        module = importlib.util.module_from_spec(spec)
        sys.modules[name] = module
        spec.loader.exec_module(module)
    return sys.modules[name]


def _resident():
    _package()
    from gbgperiodicfields_gb300 import resident
    return resident


# ------------------------------------------------------------------ cases


def listed():
    return [
        # a handful of probes of a small scalar field: one call's latency
        dict(name="probe_f64_64", kind="gather", nx=64, ny=64, nz=64, rank=0, points=257, width=4,
             dtype="f64", clustered=False, ordered=False),
        # the small drop-in deposit: 64^3 scalar field, 1e5 points, cubic
        dict(name="deposit_f64_64", kind="scatter", nx=64, ny=64, nz=64, rank=0, points=100_000, width=4,
             dtype="f64", clustered=False, scaled=False),
        # a velocity field sampled in FP64 at 1e7 partly clustered particles, quintic, in traversal order
        dict(name="gather_f64_256", kind="gather", nx=256, ny=256, nz=256, rank=1, points=10_000_000, width=6,
             dtype="f64", clustered=True, ordered=True),
        # its adjoint, cubic, added to a scaled field
        dict(name="scatter_f64_256", kind="scatter", nx=256, ny=256, nz=256, rank=1, points=10_000_000, width=4,
             dtype="f64", clustered=True, scaled=True),
        # moved points: the traversal order rebuilt, then a single-precision tensor gather on a ragged grid
        dict(name="order_f32_ragged", kind="order", nx=193, ny=160, nz=127, rank=2, points=3_000_001, width=4,
             dtype="f32", clustered=True),
        # the resident form at scale: 3 velocity and 9 gradient components, particles kept in cell order
        dict(name="step_512c12", kind="step", nx=512, ny=512, nz=512, ncomp=12, points=32_000_000, width=4,
             dtype="f64", clustered=False, sorted=True, brick="15x8x8"),
        # an ordinary resident step: one vector field, quintic, particles in no order
        dict(name="step_128c3", kind="step", nx=128, ny=128, nz=128, ncomp=3, points=500_000, width=6,
             dtype="f64", clustered=False, sorted=False, brick=""),
        # tracers in a velocity field that a solver has just advanced
        dict(name="track_256c3", kind="track", nx=256, ny=256, nz=256, ncomp=3, points=4_000_000, width=6,
             dtype="f64", clustered=True),
        # an ensemble of uneven instances replayed from a graph
        dict(name="batch_24", kind="batch", count=24, mix=7, largest=256, points=1_000_000),
        # gathers and deposits arriving together at resident fields
        dict(name="served_16", kind="served", requests=16, mix=9, largest=256, points=2_000_000),
        # a spectral field sampled at particles, FP64 at tolerance 1e-6
        dict(name="nufft2_f64_128", kind="nufft2", nx=128, ny=128, nz=128, rank=1, points=2_000_000,
             tolerance=1e-6, dtype="f64"),
        # particles deposited into spectral representation, FP32 at tolerance 1e-4
        dict(name="nufft1_f32_128", kind="nufft1", nx=128, ny=128, nz=128, rank=1, points=2_000_000,
             tolerance=1e-4, dtype="f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _axes(rng, lo, hi):
    """Three axis lengths around one size in [lo, hi]: a cube, or axes of their own, odd ones among them."""
    n = _log(rng, lo, hi)
    if rng.random() < 0.3:
        return n, n, n
    return tuple(min(hi, max(lo, int(round(n * rng.choice([0.5, 0.75, 1.0, 1.0, 1.25]))) + rng.randint(-3, 3)))
                 for _ in range(3))


def draw(rng: random.Random):
    kind = rng.choice(["gather", "gather", "scatter", "scatter", "order", "step", "step", "step", "track", "batch",
                       "served", "nufft2", "nufft1"])
    dtype = rng.choice(["f64", "f64", "f32"])
    if kind in ("gather", "scatter", "order"):
        nx, ny, nz = _axes(rng, 32, 256)
        rank = rng.choice([0, 1, 1, 2])
        width = rng.choice([4, 4, 6, 8] if kind != "scatter" else [4, 4, 6])
        # no more stencil work than the listed scatter's (FP64), and no fewer points than a few probes
        most = min(10_000_000, int(10_000_000 * 3 * 64 / (3 ** rank * width ** 3)))
        case = dict(kind=kind, nx=nx, ny=ny, nz=nz, rank=rank, points=_log(rng, 200 if kind == "gather" else 1000, most),
                    width=width, dtype=dtype, clustered=rng.random() < 0.5)
        if kind == "gather":
            case["ordered"] = rng.random() < 0.5
        if kind == "scatter":
            case["scaled"] = rng.random() < 0.5
        return case
    if kind == "step":
        nx, ny, nz = _axes(rng, 32, 384)
        ncomp, width = rng.choice([1, 3, 3, 9, 12]), rng.choice([4, 4, 6])
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, ncomp=ncomp, points=_log(rng, 2000, 8_000_000), width=width,
                    dtype=dtype, clustered=rng.random() < 0.4, sorted=rng.random() < 0.5, brick="")
    if kind == "track":
        nx, ny, nz = _axes(rng, 32, 320)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, ncomp=rng.choice([1, 3, 3, 9]), points=_log(rng, 2000, 8_000_000),
                    width=rng.choice([4, 6, 6]), dtype=dtype, clustered=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(8, 28), mix=rng.randint(100, 999999), largest=rng.choice([128, 256]),
                    points=_log(rng, 100_000, 1_000_000))
    if kind == "served":
        return dict(kind=kind, requests=rng.randint(8, 24), mix=rng.randint(100, 999999),
                    largest=rng.choice([128, 192, 256]), points=_log(rng, 200_000, 2_000_000))
    nx, ny, nz = _axes(rng, 24, 128)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, rank=rng.choice([0, 1, 1]), points=_log(rng, 5000, 2_000_000),
                tolerance=rng.choice([1e-4, 1e-6]) if dtype == "f64" else rng.choice([1e-3, 1e-4]), dtype=dtype)


# ------------------------------------------------------------------ inputs


def _dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _generator(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * int(seed) + salt)
    return g


def _colmajor(shape, dtype):
    rev = tuple(range(len(shape) - 1, -1, -1))
    return torch.empty(tuple(reversed(shape)), dtype=dtype, device="cuda").permute(rev)


def _smooth(gen, n, ncomp, dtype):
    """A real periodic field (Nx, Ny, Nz, C), column-major, of unit RMS: random modes |k| <= 24 with amplitudes
    falling as |k|^(-11/6) and random phases."""
    nx, ny, nz = n
    kx = torch.fft.fftfreq(nx, 1.0 / nx, device="cuda")[None, None, :]
    ky = torch.fft.fftfreq(ny, 1.0 / ny, device="cuda")[None, :, None]
    kz = torch.fft.rfftfreq(nz, 1.0 / nz, device="cuda")[:, None, None]
    # stored (z, y, x); the transform's half axis is z, put last for it
    k = torch.sqrt(kx * kx + ky * ky + kz * kz)
    amp = torch.where((k > 0) & (k <= 24), k.clamp_min(1) ** (-11.0 / 6.0), torch.zeros_like(k)).to(dtype)
    out = torch.empty((ncomp, nz, ny, nx), dtype=dtype, device="cuda")
    for c in range(ncomp):
        spec = torch.view_as_complex(torch.randn(amp.shape + (2,), generator=gen, device="cuda", dtype=dtype) * amp[..., None])
        real = torch.fft.irfftn(spec, s=(ny, nx, nz), dim=(1, 2, 0))
        out[c] = real / real.square().mean().sqrt()
        del spec, real
    return out.permute(3, 2, 1, 0)


def _points(gen, m, dtype, clustered):
    """(M, 3) positions in the box, column-major: uniform, or 70% uniform and 30% in 1000 Gaussian blobs."""
    pos = torch.rand((3, m), generator=gen, device="cuda", dtype=torch.float64) * TWO_PI
    if clustered:
        centres = torch.rand((3, 1000), generator=gen, device="cuda", dtype=torch.float64) * TWO_PI
        which = torch.randint(0, 1000, (m,), generator=gen, device="cuda")
        blob = centres[:, which] + 0.05 * torch.randn((3, m), generator=gen, device="cuda", dtype=torch.float64)
        inside = torch.rand((m,), generator=gen, device="cuda") < 0.3
        pos = torch.where(inside[None, :], torch.remainder(blob, TWO_PI), pos)
    return pos.to(dtype).permute(1, 0)


def _normal(gen, m, ncomp, dtype):
    return torch.randn((ncomp, m), generator=gen, device="cuda", dtype=dtype).permute(1, 0)


def _shaped(t, rank):
    """(M, 3^R) -> (M, 3, ..., 3), first tensor index fastest, column-major."""
    m = t.shape[0]
    flat = t.permute(1, 0)
    return flat.reshape((3,) * rank + (m,)).permute(tuple(range(rank, -1, -1)))


def _shaped_field(f, rank):
    n = f.shape[:3]
    flat = f.permute(3, 2, 1, 0)
    return flat.reshape((3,) * rank + (n[2], n[1], n[0])).permute(tuple(range(rank + 2, -1, -1)))


def _cell_order(pos, n):
    """Particles in the order that a cell-binned loop keeps them: by block of 8^3 cells, then by cell."""
    c = [(pos[:, d].double() * (n[d] / TWO_PI)).long().clamp_(0, n[d] - 1) for d in range(3)]
    nb = [-(-v // 8) for v in n]
    block = ((c[2] // 8) * nb[1] + c[1] // 8) * nb[0] + c[0] // 8
    key = block * 512 + ((c[2] % 8) * 8 + c[1] % 8) * 8 + c[0] % 8
    return torch.argsort(key, stable=True)


def _sizes(case):
    return case["nx"], case["ny"], case["nz"]


def _scheme(width):
    gbg = _package()
    return gbg.CatmullRom if width == 4 else gbg.LalescuSpline(width)


def _transfer_inputs(case, seed):
    """A drop-in transfer's arrays: (grid values, positions, quantities) as plain tensors."""
    gen, T, c = _generator(seed), _dtype(case), 3 ** case["rank"]
    n, m = _sizes(case), case["points"]
    data = _smooth(gen, n, c, T)
    pos = _points(gen, m, T, case["clustered"])
    q = _normal(gen, m, c, T) if case["kind"] == "scatter" else None
    return data, pos, q


def _resident_inputs(case, seed):
    gen, T = _generator(seed), _dtype(case)
    n, m, c = _sizes(case), case["points"], case["ncomp"]
    data = _smooth(gen, n, c, torch.float32)
    pos = _points(gen, m, T, case["clustered"])
    if case.get("sorted"):
        pos = pos[_cell_order(pos, n)].permute(1, 0).contiguous().permute(1, 0)
    q = _normal(gen, m, c, torch.float32)
    return data, pos, q


def _track_inputs(case, seed):
    gen, T = _generator(seed), _dtype(case)
    n, m, c = _sizes(case), case["points"], case["ncomp"]
    data = _smooth(gen, n, c, torch.float32)
    pos = _points(gen, m, T, case["clustered"])
    v1, v2 = _normal(gen, m, 3, T), _normal(gen, m, 3, T)
    return data, pos, v1, v2


# two-stage time step of the tracers: x + dt (3/2 v_n - 1/2 v_(n-1))
TERMS = (0.015, -0.005)


def _batch_mix(case):
    """The instances' grids, components, point counts and widths: part of the case, not of the seed."""
    rng = random.Random(case["mix"])
    grids = [n for n in (32, 64, 128, 256) if n <= case["largest"]]
    mix = []
    for _ in range(case["count"]):
        n = rng.choice(grids)
        mix.append(dict(nx=n, ny=n, nz=n, ncomp=rng.choice([1, 3, 9]), points=_log(rng, 1000, case["points"]),
                        width=rng.choice([4, 6]), dtype="f64", clustered=False))
    return mix


def _served_mix(case):
    """The resident fields' sizes and the requests (field, points, deposit) in their order of arrival."""
    rng = random.Random(case["mix"])
    fields = [case["largest"], max(64, case["largest"] * 3 // 4), max(64, case["largest"] // 2)]
    return fields, [(rng.randrange(3), _log(rng, 10_000, case["points"]), rng.random() < 0.3)
                    for _ in range(case["requests"])]


def _served_inputs(case, seed):
    sizes, requests = _served_mix(case)
    gen = _generator(seed)
    fields = [_smooth(gen, (n, n, n), 3, torch.float32) for n in sizes]
    return fields, [(f, _points(gen, m, torch.float64, False), _normal(gen, m, 3, torch.float32) if deposit else None)
                    for f, m, deposit in requests]


def _nufft_inputs(case, seed):
    """A band-limited spectral field (half axis x), positions and quantities."""
    gen, T = _generator(seed), _dtype(case)
    n, m, c = _sizes(case), case["points"], 3 ** case["rank"]
    phys = _smooth(gen, n, c, T)
    pos = _points(gen, m, T, False)
    q = _normal(gen, m, c, T) if case["kind"] == "nufft1" else None
    return phys, pos, q


# ------------------------------------------------------------------ the framework's side


def prepare(case, seed):
    gbg, kind = _package(), case["kind"]
    if kind in ("gather", "scatter", "order"):
        T, rank = _dtype(case), case["rank"]
        data, pos, q = _transfer_inputs(case, seed)
        grid = gbg.Grid3D(_sizes(case), (TWO_PI,) * 3, dtype=T)
        field = gbg.AbstractFieldPhysical(_shaped_field(data, rank), grid, rank)
        points = gbg.PointSet(pos)
        state = dict(kind=kind, grid=grid, field=field, points=points, scheme=_scheme(case["width"]))
        if kind == "scatter":
            state["q"] = gbg.AbstractPointValues(_shaped(q, rank), rank)
            state["scale"] = (0.5, 0.25) if case["scaled"] else (None, None)
            return state
        state["out"] = gbg.AbstractPointValues(_colmajor((case["points"],) + (3,) * rank, T), rank)
        state["order"] = None
        if kind == "order" or case["ordered"]:
            state["order"] = gbg.point_traversal_order(grid, points)
        if kind == "order":
            state["scratch"] = gbg.PointTraversalOrderScratch(grid, points)
        return state
    if kind == "step":
        res = _resident()
        data, pos, q = _resident_inputs(case, seed)
        grid = gbg.Grid3D(_sizes(case), (TWO_PI,) * 3)
        brick = tuple(int(v) for v in case["brick"].split("x")) if case["brick"] else None
        grid = grid if case["dtype"] == "f64" else gbg.Grid3D(_sizes(case), (TWO_PI,) * 3, dtype=torch.float32)
        return dict(kind=kind, field=res.ResidentField(grid, case["ncomp"], case["width"]).load(data),
                    dest=res.ResidentField(grid, case["ncomp"], case["width"]),
                    bins=res.PointBins(grid, case["points"], brick=brick), pos=pos, q=q, scheme=_scheme(case["width"]),
                    out=_colmajor((case["points"], case["ncomp"]), torch.float32))
    if kind == "track":
        res = _resident()
        data, pos, v1, v2 = _track_inputs(case, seed)
        grid = gbg.Grid3D(_sizes(case), (TWO_PI,) * 3, dtype=_dtype(case))
        return dict(kind=kind, data=data, field=res.ResidentField(grid, case["ncomp"], case["width"]),
                    bins=res.PointBins(grid, case["points"]), pos=pos, moved=_colmajor(tuple(pos.shape), pos.dtype),
                    v1=v1, v2=v2, scheme=_scheme(case["width"]),
                    out=_colmajor((case["points"], case["ncomp"]), torch.float32))
    if kind == "batch":
        res = _resident()
        items = []
        for k, one in enumerate(_batch_mix(case)):
            data, pos, q = _resident_inputs(dict(one, kind="step"), 1000 * seed + k)
            grid = gbg.Grid3D(_sizes(one), (TWO_PI,) * 3)
            items.append(dict(field=res.ResidentField(grid, one["ncomp"], 6).load(data),
                              dest=res.ResidentField(grid, one["ncomp"], 6), pos=pos, q=q,
                              bins=res.PointBins(grid, one["points"]).build(pos), scheme=_scheme(one["width"]),
                              out=_colmajor((one["points"], one["ncomp"]), torch.float32)))
        batch = res.Batch([{k: it[k] for k in ("field", "bins", "scheme", "out", "dest", "q")} for it in items])
        state = dict(kind=kind, items=items, batch=batch)

        def step():
            res.build_bins([(it["bins"], it["pos"]) for it in items])
            batch.run()
            return [it["dest"].read(torch.float32) for it in items]

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["deposits"] = step()
        return state
    if kind == "served":
        res = _resident()
        from gbgperiodicfields_gb300 import serving
        fields, requests = _served_inputs(case, seed)
        held = []
        for data in fields:
            grid = gbg.Grid3D(tuple(data.shape[:3]), (TWO_PI,) * 3)
            held.append(res.ResidentField(grid, 3, 4).load(data))
        return dict(kind=kind, fields=held, scheme=_scheme(4), server=serving.Server(slots=4, max_batch=8, timeout=60.0),
                    requests=[(f, pos, q, None if q is not None else _colmajor(tuple(pos.shape), torch.float32))
                              for f, pos, q in requests])
    # nufft2, nufft1
    T, rank = _dtype(case), case["rank"]
    phys, pos, q = _nufft_inputs(case, seed)
    grid = gbg.Grid3D(_sizes(case), (TWO_PI,) * 3, dtype=T)
    spectral = gbg.to_spectral(gbg.AbstractFieldPhysical(_shaped_field(phys, rank), grid, rank))
    plan = gbg.NUFFT(spectral, tolerance=case["tolerance"])
    state = dict(kind=kind, field=spectral, points=gbg.PointSet(pos), plan=plan)
    if kind == "nufft1":
        state["q"] = gbg.AbstractPointValues(_shaped(q, rank), rank)
    else:
        state["out"] = gbg.AbstractPointValues(_colmajor((case["points"],) + (3,) * rank, T), rank)
    return state


def run(state):
    gbg, kind = _package(), state["kind"]
    if kind == "gather":
        gbg.interpolate_(state["out"], state["field"], state["points"], state["scheme"], state["order"])
        return state["out"].data
    if kind == "scatter":
        alpha, beta = state["scale"]
        gbg.anterpolate_(state["field"], state["points"], state["q"], state["scheme"], alpha, beta)
        return state["field"].data
    if kind == "order":
        gbg.point_traversal_order_(state["order"], state["grid"], state["points"], state["scratch"])
        gbg.interpolate_(state["out"], state["field"], state["points"], state["scheme"], state["order"])
        return dict(order=state["order"].indices, values=state["out"].data)
    if kind == "step":
        res = _resident()
        state["bins"].build(state["pos"])
        res.interpolate_binned(state["field"], state["bins"], state["scheme"], out=state["out"])
        res.anterpolate_binned(state["dest"], state["bins"], state["scheme"], state["q"])
        return dict(values=state["out"], deposit=state["dest"].read(torch.float32))
    if kind == "track":
        res = _resident()
        state["field"].load(state["data"])
        state["bins"].build_displaced(state["moved"], state["pos"], ((TERMS[0], state["v1"]), (TERMS[1], state["v2"])))
        res.interpolate_binned(state["field"], state["bins"], state["scheme"], out=state["out"])
        return dict(positions=state["moved"], values=state["out"])
    if kind == "batch":
        state["graph"].replay()
        return dict(values=[it["out"] for it in state["items"]], deposits=state["deposits"])
    if kind == "served":
        server, tickets = state["server"], []
        for f, pos, q, out in state["requests"]:
            if q is None:
                tickets.append(server.interpolate(state["fields"][f], pos, state["scheme"], out=out))
            else:
                tickets.append(server.anterpolate(state["fields"][f], pos, state["scheme"], q, 1.0, 1.0))
        values = [server.result(t) for t in tickets]
        return dict(values=[v for v in values if v is not None],
                    fields=[f.read(torch.float32) for f in state["fields"]])
    if kind == "nufft2":
        gbg.interpolate_(state["out"], state["field"], state["points"], state["plan"])
        return state["out"].data
    gbg.anterpolate_(state["field"], state["points"], state["q"], state["plan"])
    return state["field"].data


# ------------------------------------------------------------------ the work a pass cannot do without


def _nodes(n, m, width):
    """Nodes that a gather has to read: the grid's, or the points' own stencils where those are fewer."""
    return min(n[0] * n[1] * n[2], m * width ** 3)


def _nufft_width(tolerance):
    return min(16, max(4, math.ceil(-math.log10(tolerance)) + 2))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        each = [work(dict(one, kind="step", sorted=False, brick="")) for one in _batch_mix(case)]
        return dict(bytes=sum(w["bytes"] for w in each), flops=sum(w["flops"] for w in each))
    if kind == "served":
        fields, requests = _served_mix(case)
        data = flops = 0.0
        for f, m, deposit in requests:
            n = (fields[f],) * 3
            touched = _nodes(n, m, 4)
            data += m * (24 + 12) + touched * 12 * (2 if deposit else 1)
            flops += 2.0 * m * 64 * 3
        return dict(bytes=data + sum(12.0 * n ** 3 for n in fields), flops=flops)
    n, m = _sizes(case), case["points"]
    nodes = n[0] * n[1] * n[2]
    s = 8 if case["dtype"] == "f64" else 4
    if kind in ("nufft2", "nufft1"):
        c, w = 3 ** case["rank"], _nufft_width(case["tolerance"])
        fine = 8 * nodes
        return dict(bytes=float(m * (3 + c) * s + (n[0] // 2 + 1) * n[1] * n[2] * c * 2 * s),
                    flops=2.0 * m * w ** 3 * c + 2.5 * fine * math.log2(fine) * c)
    w = case["width"]
    c = case["ncomp"] if "ncomp" in case else 3 ** case["rank"]
    flops = 2.0 * m * w ** 3 * c
    if kind == "gather":
        return dict(bytes=float(m * (3 + c) * s + _nodes(n, m, w) * c * s + (4 * m if case["ordered"] else 0)), flops=flops)
    if kind == "scatter":
        return dict(bytes=float(m * (3 + c) * s + nodes * c * s * (2 if case["scaled"] else 1)), flops=flops)
    if kind == "order":
        return dict(bytes=float(m * (3 + c) * s + _nodes(n, m, w) * c * s + 4 * m), flops=flops)
    if kind == "step":
        return dict(bytes=float(m * (3 * s + 8 * c) + (_nodes(n, m, w) + nodes) * c * 4), flops=2 * flops)
    # track: the field as given, positions and two velocities in, positions and values out
    return dict(bytes=float(nodes * c * 4 + m * (12 * s + 4 * c)), flops=flops)


# ------------------------------------------------------------------ the same in 64 bits, by plain torch


def _derivative_weights(nodes, order):
    """Finite-difference weights at 0 of the derivatives 0..order over integer nodes (Vandermonde solve)."""
    a = np.array([[float(x) ** p / math.factorial(p) for x in nodes] for p in range(len(nodes))])
    return [np.linalg.solve(a, np.eye(len(nodes))[d]) for d in range(order + 1)]


def _spline(width):
    """Coefficients [node, power] of the smooth local spline: on a cell the polynomial that matches, at both ends,
    the centred finite-difference derivatives 0..width/2-1 taken over width-1 nodes."""
    n, m = width // 2 - 1, width // 2 - 1
    weights = _derivative_weights(list(range(-n, n + 1)), m)
    powers = 2 * m + 2
    a = np.zeros((powers, powers))
    for d in range(m + 1):
        a[d, d] = math.factorial(d)
        for p in range(d, powers):
            a[m + 1 + d, p] = math.factorial(p) / math.factorial(p - d)
    hermite = np.linalg.inv(a)  # column: the polynomial with that one derivative equal to 1
    coef = np.zeros((width, powers))
    for d in range(m + 1):
        for k in range(2 * n + 1):
            coef[k] += weights[d][k] * hermite[:, d]
            coef[k + 1] += weights[d][k] * hermite[:, m + 1 + d]
    return coef


def _locate(pos, n, dtype):
    """Cell and fraction of positions on the box [0, 2 pi)^3, whose length is held in the grid's type."""
    length = float(torch.tensor(TWO_PI, dtype=dtype).double())
    u = pos.double() * (torch.tensor(n, dtype=torch.float64, device="cuda") / length)
    base = torch.floor(u)
    return base.long(), u - base


def _spline_stencil(pos, n, width, dtype):
    base, t = _locate(pos, n, dtype)
    coef = torch.from_numpy(_spline(width)).cuda()
    w = torch.zeros(pos.shape + (width,), dtype=torch.float64, device="cuda")
    for p in range(coef.shape[1] - 1, -1, -1):
        w = w * t[..., None] + coef[:, p]
    first = base - (width // 2 - 1)
    return w, first


def _window_stencil(pos, fine, width, beta, dtype):
    base, t = _locate(pos, fine, dtype)
    half = torch.where(t < 0.5, (width + 1) // 2, width // 2) if width % 2 else torch.full_like(base, width // 2)
    i = torch.arange(1, width + 1, device="cuda")
    z = 2.0 * (t[..., None] - (i - half[..., None])) / width
    w = torch.exp(beta * (torch.sqrt((1 - z * z).clamp_min(0)) - 1))
    return w, base + 1 - half


def _exact_gather(data, pos, stencil, chunk=1_000_000):
    """sum over the stencil of w f; data (Nx, Ny, Nz, C) of any layout, the result (M, C)."""
    n, c = data.shape[:3], data.shape[3]
    flat = data.permute(2, 1, 0, 3).reshape(-1, c).double()  # node-major rows, x fastest
    out = torch.empty((pos.shape[0], c), dtype=torch.float64, device="cuda")
    for a in range(0, pos.shape[0], chunk):
        w, first = stencil(pos[a:a + chunk])
        acc = torch.zeros((w.shape[0], c), dtype=torch.float64, device="cuda")
        width = w.shape[-1]
        ix = [torch.remainder(first[:, d, None] + torch.arange(width, device="cuda"), n[d]) for d in range(3)]
        for k in range(width):
            for j in range(width):
                row = (ix[2][:, k] * n[1] + ix[1][:, j]) * n[0]
                wyz = w[:, 2, k] * w[:, 1, j]
                for i in range(width):
                    acc += (wyz * w[:, 0, i])[:, None] * flat[row + ix[0][:, i]]
        out[a:a + chunk] = acc
    return out


def _exact_scatter(n, pos, q, stencil, chunk=1_000_000):
    """The adjoint: (Nx, Ny, Nz, C)."""
    c = q.shape[1]
    flat = torch.zeros((n[0] * n[1] * n[2], c), dtype=torch.float64, device="cuda")
    for a in range(0, pos.shape[0], chunk):
        w, first = stencil(pos[a:a + chunk])
        qq = q[a:a + chunk].double()
        width = w.shape[-1]
        ix = [torch.remainder(first[:, d, None] + torch.arange(width, device="cuda"), n[d]) for d in range(3)]
        for k in range(width):
            for j in range(width):
                row = (ix[2][:, k] * n[1] + ix[1][:, j]) * n[0]
                wyz = w[:, 2, k] * w[:, 1, j]
                for i in range(width):
                    flat.index_add_(0, row + ix[0][:, i], (wyz * w[:, 0, i])[:, None] * qq)
    return flat.reshape(n[2], n[1], n[0], c).permute(2, 1, 0, 3)


def _window_transform(n, stored, width, beta):
    """1 / psi_hat of the window on an axis of n modes at oversampling 2 (0 at an even axis's Nyquist mode)."""
    i = np.arange(stored)
    f = i if stored < n else np.where(i < (n + 1) // 2, i, i - n)
    omega = 2 * np.pi * f / (2.0 * n)
    theta = -np.pi / 2 + np.pi * np.arange(257) / 256
    trap = np.ones(257)
    trap[0] = trap[-1] = 0.5
    half = width / 2
    psi = half * (np.pi / 256) * np.sum(trap * np.exp(beta * (np.cos(theta) - 1))
                                        * np.cos(omega[:, None] * half * np.sin(theta)) * np.cos(theta), axis=1)
    dec = 1 / psi
    if n % 2 == 0:
        dec[stored - 1 if stored < n else n // 2] = 0.0
    return torch.from_numpy(dec).cuda()


def _shared(n, fine, half_axis):
    """Stored indices of the modes that the two grids share on one axis: (coarse, fine)."""
    if half_axis:
        k = torch.arange((n + 1) // 2, device="cuda")
        return k, k
    i = torch.cat([torch.arange((n + 1) // 2, device="cuda"), torch.arange(n - (n - n // 2 - 1), n, device="cuda")])
    return i, torch.where(i < (n + 1) // 2, i, fine - (n - i))


def _exact_nufft(case, seed):
    n, rank = _sizes(case), case["rank"]
    fine = tuple(2 * v for v in n)
    T = _dtype(case)
    width = _nufft_width(case["tolerance"])
    real = np.float32 if case["dtype"] == "f32" else np.float64
    beta = float(real(real(23) / real(10) * real(width)))
    phys, pos, q = _nufft_inputs(case, seed)
    c = 3 ** rank
    stored = (n[0] // 2 + 1, n[1], n[2])
    dec = [_window_transform(n[d], stored[d], width, beta) for d in range(3)]
    dec = dec[0][:, None, None, None] * dec[1][None, :, None, None] * dec[2][None, None, :, None]
    pairs = [_shared(n[d], fine[d], d == 0) for d in range(3)]
    ci = (pairs[0][0][:, None, None], pairs[1][0][None, :, None], pairs[2][0][None, None, :])
    fi = (pairs[0][1][:, None, None], pairs[1][1][None, :, None], pairs[2][1][None, None, :])

    def stencil(p):
        return _window_stencil(p, fine, width, beta, T)

    if case["kind"] == "nufft2":
        spec = torch.fft.rfftn(phys, dim=(1, 2, 0)).to(torch.complex128) * dec
        wide = torch.zeros((fine[0] // 2 + 1, fine[1], fine[2], c), dtype=torch.complex128, device="cuda")
        wide[fi] = spec[ci] * 8.0
        values = torch.fft.irfftn(wide, s=(fine[1], fine[2], fine[0]), dim=(1, 2, 0))
        return _shaped(_exact_gather(values, pos, stencil).permute(1, 0).contiguous().permute(1, 0), rank)
    spread = _exact_scatter(fine, pos, q, stencil)
    spec = torch.fft.rfftn(spread, dim=(1, 2, 0))
    out = torch.zeros(stored + (c,), dtype=torch.complex128, device="cuda")
    out[ci] = spec[fi]
    return _shaped_field((out * dec).permute(3, 2, 1, 0).contiguous().permute(3, 2, 1, 0), rank)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("nufft2", "nufft1"):
        return _exact_nufft(case, seed)
    if kind in ("gather", "scatter", "order"):
        data, pos, q = _transfer_inputs(case, seed)
        n, rank, T = _sizes(case), case["rank"], _dtype(case)

        def stencil(p):
            return _spline_stencil(p, n, case["width"], T)

        if kind == "scatter":
            out = _exact_scatter(n, pos, q, stencil)
            if case["scaled"]:
                out = 0.5 * out + 0.25 * data.double()
            return _shaped_field(out.permute(3, 2, 1, 0).contiguous().permute(3, 2, 1, 0), rank)
        values = _shaped(_exact_gather(data, pos, stencil).permute(1, 0).contiguous().permute(1, 0), rank)
        return dict(order=None, values=values) if kind == "order" else values
    if kind == "step":
        data, pos, q = _resident_inputs(case, seed)
        n, T = _sizes(case), _dtype(case)

        def stencil(p):
            return _spline_stencil(p, n, case["width"], T)

        values = _exact_gather(data, pos, stencil)
        del data
        return dict(values=values, deposit=_exact_scatter(n, pos, q, stencil))
    if kind == "track":
        data, pos, v1, v2 = _track_inputs(case, seed)
        n, T = _sizes(case), _dtype(case)
        length = float(torch.tensor(TWO_PI, dtype=T).double())
        a, b = (float(torch.tensor(x, dtype=T).double()) for x in TERMS)
        moved = torch.remainder(pos.double() + a * v1.double() + b * v2.double(), length)
        # the gather is of the positions as the grid's type holds them
        held = moved.to(T)

        def stencil(p):
            return _spline_stencil(p, n, case["width"], T)

        return dict(positions=moved, values=_exact_gather(data, held, stencil))
    if kind == "batch":
        values, deposits = [], []
        for k, one in enumerate(_batch_mix(case)):
            got = exact(dict(one, kind="step", sorted=False, brick=""), 1000 * seed + k)
            values.append(got["values"])
            deposits.append(got["deposit"])
        return dict(values=values, deposits=deposits)
    fields, requests = _served_inputs(case, seed)
    fields = [f.double() for f in fields]
    values = []
    for f, pos, q in requests:
        n = tuple(fields[f].shape[:3])

        def stencil(p, n=n):
            return _spline_stencil(p, n, 4, torch.float64)

        if q is None:
            values.append(_exact_gather(fields[f], pos, stencil))
        else:
            fields[f] = fields[f] + _exact_scatter(n, pos, q, stencil)
    return dict(values=values, fields=fields)
