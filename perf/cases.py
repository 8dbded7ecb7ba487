"""The work that users of this framework have it do, as timed cases.

A case names one kind of work (``kind``) and its sizes and options:

- ``curves``: recording rounds on host arrays, ``dpa_advect_round`` with a sink
  that stores the curves in the program's own arrays: the drop-in for the
  reference's advection stage. Sizes run from an interactive handful of seeds
  to rounds whose curves take hundreds of megabytes.
- ``round``: ``ParticleAdvector.advect`` on host arrays, end positions only.
- ``device``: ``dpa_advect_device`` on device arrays, end positions only: a
  program that keeps its particles on the GPU.
- ``batch``: ``dpa_advect_batch_device``, many seed sets of uneven size and
  iteration count in one launch, with each set's step count.
- ``ftle``: lattice seeding, advection and FTLE on the device.
- ``ftle_field``: the FTLE stage alone, of a given flow map.
- ``pathlines``: ``advect_pathlines`` through a time-varying field.
- ``serve``: a burst of mixed requests to the request server, until the last
  one is back.
- ``insitu``: a simulation's new time step: its field is made resident,
  sampled by a few steps of the particles, and let go.

Fields are synthetic: ABC flow, the double gyre, or the curl of smoothed
noise, all made on the GPU from the seed.
"""
import ctypes as C
import functools
import math
import random

import numpy as np
import torch

from dpa_b200 import (Context, Field, ParticleAdvector, Particles, RegularGrid, advect_pathlines,
                      fields, seeds)
from dpa_b200 import _native as N
from dpa_b200.serve import Server


def listed():
    return [
        # A user looking at a flow: a hundred streamlines through a small
        # field, recorded. Launches, copies and host work are all there is.
        {"name": "curves_small", "kind": "curves", "field": "abc", "n0": 32, "n1": 32, "n2": 32,
         "h": 2 * math.pi / 31, "storage": "f32", "integrator": "runge_kutta_4", "seeds": 100,
         "iterations": 50, "step": 0.02, "per_round": 100},
        # The plain method's configuration: 4096 recorded seeds in ABC flow.
        {"name": "curves_4k", "kind": "curves", "field": "abc", "n0": 64, "n1": 64, "n2": 64,
         "h": 2 * math.pi / 63, "storage": "f32", "integrator": "runge_kutta_4", "seeds": 4096,
         "iterations": 1000, "step": 0.01, "per_round": 4096},
        # Dense integral curves in several rounds; an odd seed count leaves a
        # ragged last round.
        {"name": "curves_large", "kind": "curves", "field": "curl", "n0": 128, "n1": 128,
         "n2": 128, "h": 1.0, "storage": "f32", "integrator": "runge_kutta_4", "seeds": 40001,
         "iterations": 300, "step": 0.25, "per_round": 16384},
        # A round without recording from and to host arrays, on an uneven grid
        # whose spacing is no power of two.
        {"name": "round_end", "kind": "round", "field": "curl", "n0": 160, "n1": 96, "n2": 129,
         "h": 0.7, "storage": "f32", "integrator": "runge_kutta_4", "seeds": 262147,
         "iterations": 300, "step": 0.175, "per_round": 262147},
        # The throughput configuration.
        {"name": "device_f32", "kind": "device", "field": "curl", "n0": 256, "n1": 256, "n2": 256,
         "h": 1.0, "storage": "f32", "integrator": "runge_kutta_4", "seeds": 1048576,
         "iterations": 2000, "step": 0.25},
        # The half-precision field of a mid-sized call, odd sizes.
        {"name": "device_f16", "kind": "device", "field": "curl", "n0": 192, "n1": 255, "n2": 161,
         "h": 1.0, "storage": "f16", "integrator": "runge_kutta_4", "seeds": 200003,
         "iterations": 400, "step": 0.25},
        # The large, batched configuration: 64 uneven seed sets, 512^3 nodes.
        {"name": "batch_f32", "kind": "batch", "field": "curl", "n0": 512, "n1": 512, "n2": 512,
         "h": 1.0, "storage": "f32", "integrator": "runge_kutta_4", "sets": 64,
         "seeds": 16777216, "least": 200, "iterations": 4000, "step": 0.25},
        # The FTLE configuration: every second node of a 256^3 field seeded.
        {"name": "ftle_lattice", "kind": "ftle", "field": "abc", "n0": 256, "n1": 256, "n2": 256,
         "h": 2 * math.pi / 255, "storage": "f32_edges", "integrator": "runge_kutta_4",
         "stride": 2, "iterations": 250, "step": 0.02},
        # FTLE of a flow map that a program already holds.
        {"name": "ftle_field", "kind": "ftle_field", "n0": 256, "n1": 192, "n2": 250, "h": 1.0,
         "stride": 2, "mapping": "lattice", "iterations": 200, "step": 0.25},
        # Pathlines through 32 time slices, from and to host arrays.
        {"name": "pathlines", "kind": "pathlines", "n0": 128, "n1": 64, "n2": 64, "slices": 32,
         "storage": "f32", "integrator": "runge_kutta_4", "seeds": 250000, "iterations": 1000,
         "step": 0.005},
        # A burst of requests at the server: end positions, recordings,
        # pathlines and FTLE in one mix, half-precision fields.
        {"name": "serve_burst", "kind": "serve", "n0": 128, "n1": 128, "n2": 128,
         "storage": "f16", "requests": 12, "most_seeds": 100000, "most_iterations": 1500},
        # One time step of a coupled simulation.
        {"name": "insitu", "kind": "insitu", "field": "curl", "n0": 192, "n1": 192, "n2": 192,
         "h": 1.0, "storage": "f32", "integrator": "euler", "seeds": 50000, "iterations": 10,
         "step": 0.25},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(lo, hi):
        return {"n0": log_int(lo, hi), "n1": log_int(lo, hi), "n2": log_int(lo, hi)}

    storage = rng.choice(["f32", "f32", "f16", "bf16", "f32_edges"])
    integrator = rng.choice(["runge_kutta_4"] * 4 + ["euler", "runge_kutta_4_true",
                            "runge_kutta_dormand_prince_5", "runge_kutta_cash_karp_54",
                            "modified_midpoint"])
    h = rng.choice([1.0, 0.5, 0.7, 0.1])
    kind = rng.choice(["curves"] * 3 + ["device"] * 4 + ["round", "batch", "ftle", "ftle_field",
                                                         "pathlines", "serve", "insitu"])
    flow = {"kind": kind, "field": "curl", "h": h, "storage": storage, "integrator": integrator,
            "step": h * rng.choice([0.1, 0.2, 0.25, 0.5])}
    if kind in ("curves", "round"):
        n = log_int(50, 60000 if kind == "curves" else 400000)
        most = max(21, min(1500, (12_000_000 if kind == "curves" else 200_000_000) // n))
        return {**flow, **grid(24, 160), "seeds": n, "iterations": log_int(20, most),
                "per_round": rng.choice([n, max(1, n // 2 + 1)])}
    if kind == "device":
        return {**flow, **grid(32, 256), "seeds": log_int(1000, 1000000),
                "iterations": log_int(50, 1500)}
    if kind == "batch":
        return {**flow, **grid(64, 320), "sets": rng.randint(2, 64),
                "seeds": log_int(100000, 4000000), "least": rng.randint(20, 200),
                "iterations": log_int(250, 2000)}
    if kind == "ftle":
        return {**flow, **grid(48, 200), "stride": rng.choice([1, 2]),
                "iterations": log_int(20, 250)}
    if kind == "ftle_field":
        return {"kind": kind, **grid(40, 256), "h": h, "stride": 2,
                "mapping": rng.choice(["lattice", "reference"]),
                "iterations": log_int(20, 400), "step": flow["step"]}
    if kind == "pathlines":
        return {"kind": kind, **grid(24, 128), "slices": rng.randint(4, 32), "storage": storage,
                "integrator": rng.choice(["runge_kutta_4", "euler", "runge_kutta_4_true"]),
                "seeds": log_int(500, 400000), "iterations": log_int(50, 1000),
                "step": rng.choice([0.005, 0.004, 0.0025])}
    if kind == "serve":
        return {"kind": kind, **grid(48, 160), "storage": rng.choice(["f16", "f32"]),
                "requests": rng.randint(2, 12), "most_seeds": log_int(2000, 100000),
                "most_iterations": log_int(200, 1500)}
    return {**flow, **grid(48, 256), "seeds": log_int(500, 300000),
            "iterations": rng.randint(1, 40)}


# Inputs ---------------------------------------------------------------------


def _shape(case):
    return case["n0"], case["n1"], case["n2"]


def _generator(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 16 + salt)
    return g


def _curl(shape, seed, sigma):
    """The curl of a vector potential of Gaussian-smoothed noise, unit RMS
    speed, components stored in the reference's reversed order."""
    g = _generator(seed)
    f = [torch.fft.fftfreq(n, device="cuda") for n in shape[:2]]
    f.append(torch.fft.rfftfreq(shape[2], device="cuda"))
    e = [torch.exp(-0.5 * (2 * math.pi * sigma * x) ** 2) for x in f]
    psi = []
    for _ in range(3):
        spectrum = torch.fft.rfftn(torch.randn(shape, generator=g, device="cuda"))
        spectrum *= e[0][:, None, None] * e[1][None, :, None] * e[2][None, None, :]
        psi.append(torch.fft.irfftn(spectrum, s=shape))
        del spectrum

    def d(a, axis):
        return torch.roll(a, -1, axis) - torch.roll(a, 1, axis)

    out = torch.empty(tuple(shape) + (3,), device="cuda")
    out[..., 2] = d(psi[2], 1) - d(psi[1], 2)
    out[..., 1] = d(psi[0], 2) - d(psi[2], 0)
    out[..., 0] = d(psi[1], 0) - d(psi[0], 1)
    out /= torch.sqrt(3 * torch.mean(out * out))
    return out


def _abc(shape, h, seed):
    """ABC flow, its phases drawn from the seed."""
    p = torch.rand(3, generator=_generator(seed), device="cuda", dtype=torch.float64).tolist()
    x, y, z = torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float64) * h + 6 * q
                               for n, q in zip(shape, p)], indexing="ij")
    a, b, c = fields.ABC_A, fields.ABC_B, fields.ABC_C
    u = (a * torch.sin(z) + c * torch.cos(y), b * torch.sin(x) + a * torch.cos(z),
         c * torch.sin(y) + b * torch.cos(x))
    return torch.stack([u[2], u[1], u[0]], dim=-1).float()


def _data(case, seed):
    shape = _shape(case)
    if case.get("field") == "abc":
        return _abc(shape, float(np.float32(case["h"])), seed)
    return _curl(shape, seed, 8.0 if max(shape) > 400 else 4.0)


def _grid(data, h):
    shape = tuple(data.shape[:3])
    spacing = np.full(3, h, np.float32)
    return RegularGrid(data, np.zeros(3, np.float32), np.array(shape, np.float32) * spacing,
                       spacing)


def _seeds(case, seed, count):
    """Seeds uniform in the valid domain, on the device."""
    u = torch.rand((count, 3), generator=_generator(seed, 1), device="cuda")
    top = [(n - 1) * float(np.float32(case["h"])) for n in _shape(case)]
    return u * torch.tensor(top, device="cuda", dtype=torch.float32)


@functools.lru_cache(maxsize=2)
def _gyre(shape, slices):
    """The double gyre has no random part."""
    return fields.double_gyre(shape, slices)


def _set_plan(case):
    """Sizes (log-uniform, scaled to the case's total) and iteration counts of
    a batch's seed sets; the sets of a case do not depend on the seed."""
    rng = random.Random(case["sets"])
    raw = [math.exp(rng.uniform(math.log(1e3), math.log(1e6))) for _ in range(case["sets"])]
    scale = case["seeds"] / sum(raw)
    sizes = [max(1, int(r * scale)) for r in raw]
    return sizes, [rng.randint(case["least"], case["iterations"]) for _ in sizes]


def _request_plan(case):
    """(what, seeds, iterations, recorded) of each request, independent of the
    seed. Half of them record: pathlines, which never leave the gyre."""
    rng = random.Random(case["requests"])
    plan = []
    for i in range(case["requests"]):
        what = "ftle" if i % 10 == 7 else "curl" if i % 2 else "pathlines"
        record = what == "pathlines"
        most = min(case["most_seeds"], 4000 if record else case["most_seeds"])
        n = int(math.exp(rng.uniform(math.log(100), math.log(max(101, most)))))
        plan.append((what, n, rng.randint(100, max(101, case["most_iterations"])), record))
    return plan


def _pointer(t):
    return C.c_void_p(t.data_ptr())


class _State:
    """What a user's program holds; closes what it opened, server first."""

    server = None

    def __del__(self):
        if self.server is not None:
            self.server.close()


def _device_particles(s, pos, rem):
    s.seeds, s.iterations = pos, rem
    s.pos, s.rem = torch.empty_like(pos), torch.empty_like(rem)
    s.term = torch.empty(pos.shape[0], dtype=torch.uint8, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    s = _State()
    s.case = case
    s.ctx = Context(0)
    s.stream = torch.cuda.ExternalStream(s.ctx.stream)
    if kind != "pathlines" and kind != "serve" and kind != "ftle_field":
        data = _data(case, seed)
        s.grid = _grid(data, case["h"])
        torch.cuda.synchronize()
        if kind == "insitu":
            s.data = data
        else:
            s.field = Field(s.ctx, s.grid, case["storage"], device_pointer=data.data_ptr())
        s.options = N.AdvectOptions(N.INTEGRATORS[case["integrator"]],
                                    float(np.float32(case["step"])), 0, 0, 0, 1, 0)
    if kind == "round":
        n = case["seeds"]
        s.particles = Particles.create(_seeds(case, seed, n).cpu().numpy(), case["iterations"])
        s.advector = ParticleAdvector(s.ctx, case["per_round"], "none", case["integrator"],
                                      case["step"], False, False)
        s.grid.data = s.grid.data[:1, :1, :1]  # the field is resident
    elif kind == "curves":
        n = case["seeds"]
        s.particles = Particles.create(_seeds(case, seed, n).cpu().numpy(), case["iterations"])
        s.grid.data = s.grid.data[:1, :1, :1]
        s.options.record, s.options.colors = 1, 1
        s.options.index64 = int(case["per_round"] * case["iterations"] > 0xFFFFFFFF)
        s.position, s.remaining = np.empty((n, 3), np.float32), np.empty(n, np.uint64)
        s.termination = np.zeros(n, np.uint8)
        # Room for every particle's whole curve; what a round does not need
        # stays zero.
        room = n * (case["iterations"] + 2)
        s.vertices, s.colors = np.zeros((room, 3), np.float32), np.zeros(room, np.float32)
        s.indices = np.zeros(2 * room, np.uint64 if s.options.index64 else np.uint32)
        s.sink = N.CURVE_SINK(functools.partial(_store_chunk, s))
    elif kind in ("device", "insitu"):
        n = case["seeds"]
        _device_particles(s, _seeds(case, seed, n),
                          torch.full((n,), case["iterations"], dtype=torch.int64, device="cuda"))
    elif kind == "batch":
        sizes, iterations = _set_plan(case)
        rem = torch.repeat_interleave(torch.tensor(iterations), torch.tensor(sizes)).cuda()
        _device_particles(s, _seeds(case, seed, sum(sizes)), rem)
        s.offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
        s.steps = np.zeros(len(sizes), np.uint64)
    elif kind == "ftle":
        n = _lattice(s, None)
        _device_particles(s, torch.empty((n, 3), device="cuda"),
                          torch.full((n,), case["iterations"], dtype=torch.int64, device="cuda"))
        s.ftle = torch.empty(tuple(n // case["stride"] for n in _shape(case)), device="cuda")
    elif kind == "ftle_field":
        data = torch.zeros(_shape(case) + (3,), device="cuda")
        s.grid = _grid(data, case["h"])
        s.field = Field(s.ctx, s.grid, "f32", device_pointer=data.data_ptr())
        s.seeds, s.pos = _flow_map(case, seed)
        s.ftle = torch.empty(s.seeds.shape[:3], device="cuda")
    elif kind == "pathlines":
        gyre = _gyre(_shape(case), case["slices"])
        s.field = s.ctx.field(gyre, case["storage"])
        s.positions, s.times = _pathline_starts(case["seeds"], seed)
    else:
        data = _curl(_shape(case), seed, 4.0)
        torch.cuda.synchronize()
        s.curl = Field(s.ctx, _grid(data, 1.0), case["storage"], device_pointer=data.data_ptr())
        s.gyre = s.ctx.field(_gyre((64, 32, 32), 16), case["storage"])
        s.server = Server(s.ctx, particle_capacity=2_000_000, vertex_capacity=80_000_000,
                          steps_per_tick=64, max_requests=64, reserved_percent=10)
        s.ids = {"curl": s.server.add_field(s.curl), "pathlines": s.server.add_field(s.gyre)}
        s.requests = []
        box = {**case, "h": 1.0}
        for i, (what, n, iterations, record) in enumerate(_request_plan(case)):
            start = 0.0
            if what == "pathlines":
                pos, t = _pathline_starts(n, seed * 64 + i)
                start = 0.5 * float(t[0])
            elif what == "ftle":
                pos = seeds.generate(np.zeros(3, np.float32),
                                     np.array(_shape(case), np.float32), (4.0, 4.0, 4.0),
                                     iterations).position
            else:
                pos = _seeds(box, seed * 64 + i, n).cpu().numpy()
            s.requests.append((what, pos, iterations, record, start))
    torch.cuda.synchronize()
    return s


def _pathline_starts(count, seed):
    u = torch.rand((count, 4), generator=_generator(seed, 1), device="cuda").cpu().numpy()
    return (u[:, :3] * np.array([2.0, 1.0, 1.0], np.float32)).astype(np.float32), \
        (u[:, 3] * np.float32(4.0)).astype(np.float32)


def _flow_map(case, seed):
    """A lattice of seeds and where a smooth random deformation takes them."""
    shape = tuple(n // case["stride"] for n in _shape(case))
    h = float(np.float32(case["h"])) * case["stride"]
    axes = [torch.arange(n, device="cuda", dtype=torch.float32) * h for n in shape]
    x = torch.stack(torch.meshgrid(*axes, indexing="ij"), dim=-1)
    r = torch.rand((3, 4, 5), generator=_generator(seed, 2), device="cuda")
    out = x.clone()
    for c in range(3):
        for k in r[c]:
            wave = (k[:3] * 2 - 1) * (0.5 / h)
            out[..., c] += (3.0 * h * k[3]) * torch.sin(x @ wave + 6.2831853 * k[4])
    return x.contiguous(), out.contiguous()


# Passes ---------------------------------------------------------------------


def run(s):
    return _RUN[s.case["kind"]](s)


def _run_round(s):
    p = s.advector.advect(s.field, s.particles).inactive_particles
    return {"position": p.position, "remaining": p.remaining_iterations,
            "termination": p.termination}


def _store_chunk(s, user, chunk):
    c = chunk.contents
    v, i = s.first_vertex + c.vertex_offset, s.first_index + c.index_offset
    C.memmove(s.vertices.ctypes.data + 12 * v, c.vertices, 12 * c.vertex_count)
    C.memmove(s.colors.ctypes.data + 4 * v, c.colors, 4 * c.vertex_count)
    size = s.indices.itemsize
    if c.index_count:
        C.memmove(s.indices.ctypes.data + size * i, c.indices, size * c.index_count)
    s.vertex_count = c.vertex_offset + c.vertex_count
    s.index_count = c.index_offset + c.index_count
    return 0


def _host(a, first):
    return C.c_void_p(a.ctypes.data + first * a.strides[0])


def _run_curves(s):
    """Rounds from the tail of the particles, as the reference takes them."""
    s.position[:] = s.particles.position
    s.remaining[:] = s.particles.remaining_iterations
    s.first_vertex = s.first_index = 0
    end, rounds = s.case["seeds"], []
    while end > 0:
        begin = max(0, end - s.case["per_round"])
        s.vertex_count = s.index_count = 0
        s.ctx.check(s.ctx._lib.dpa_advect_round(
            s.ctx.handle, s.field.handle, C.byref(s.options), end - begin,
            _host(s.position, begin), _host(s.remaining, begin), _host(s.termination, begin),
            s.sink, None))
        s.first_vertex += s.vertex_count
        s.first_index += s.index_count
        rounds.append((s.vertex_count, s.index_count))
        end = begin
    return {"position": s.position, "remaining": s.remaining, "termination": s.termination,
            "vertices": s.vertices, "colors": s.colors, "indices": s.indices, "rounds": rounds}


def _reset(s):
    with torch.cuda.stream(s.stream):
        s.pos.copy_(s.seeds)
        s.rem.copy_(s.iterations)


def _advect(s, field):
    s.ctx.check(s.ctx._lib.dpa_advect_device(
        s.ctx.handle, field.handle, C.byref(s.options), s.pos.shape[0], _pointer(s.pos),
        _pointer(s.rem), _pointer(s.term), None))


def _ends(s):
    return {"position": s.pos, "remaining": s.rem, "termination": s.term}


def _run_device(s):
    _reset(s)
    _advect(s, s.field)
    return _ends(s)


def _run_insitu(s):
    field = Field(s.ctx, s.grid, s.case["storage"], device_pointer=s.data.data_ptr())
    _reset(s)
    _advect(s, field)
    field.close()
    return _ends(s)


def _run_batch(s):
    _reset(s)
    s.ctx.check(s.ctx._lib.dpa_advect_batch_device(
        s.ctx.handle, s.field.handle, C.byref(s.options), len(s.steps),
        s.offsets.ctypes.data_as(N._U64P), _pointer(s.pos), _pointer(s.rem), _pointer(s.term),
        s.steps.ctypes.data_as(N._U64P), None))
    return {**_ends(s), "steps": s.steps.astype(np.int64)}


def _f3(values):
    return (C.c_float * 3)(*[float(v) for v in values])


def _estimate(s, n, original, final, mapping):
    stride = _f3([s.case["stride"]] * 3)
    s.ctx.check(s.ctx._lib.dpa_ftle_estimate_device(
        s.ctx.handle, s.field.handle, stride, s.case["iterations"],
        float(np.float32(s.case["step"])), n, _pointer(original), _pointer(final),
        N.FTLE_MAPPING[mapping], _pointer(s.ftle), None, None))


def _lattice(s, out):
    """Writes the seed lattice to `out` (None: nothing); returns its size."""
    n = C.c_uint64()
    stride = _f3([float(np.float32(s.case["h"])) * s.case["stride"]] * 3)
    s.ctx.check(s.ctx._lib.dpa_seed_lattice_device(
        s.ctx.handle, _f3(s.grid.offset), _f3(s.grid.size), stride, None, C.byref(n), None,
        None if out is None else _pointer(out), None))
    return n.value


def _run_ftle(s):
    n = _lattice(s, s.seeds)
    _reset(s)
    _advect(s, s.field)
    _estimate(s, n, s.seeds, s.pos, "reference")
    return {**_ends(s), "ftle": s.ftle}


def _run_ftle_field(s):
    _estimate(s, s.ftle.numel(), s.seeds, s.pos, s.case["mapping"])
    return s.ftle


def _run_pathlines(s):
    c = s.case
    out = advect_pathlines(s.ctx, s.field, s.positions, s.times, c["iterations"],
                           c["integrator"], c["step"])
    return {"position": out.position, "time": out.time, "remaining": out.remaining_iterations,
            "termination": out.termination}


def _run_serve(s):
    ids = []
    for what, pos, iterations, record, start in s.requests:
        gyre = what == "pathlines"
        ids.append(s.server.submit(s.ids["pathlines" if gyre else "curl"], pos, iterations,
                                   "runge_kutta_4", 0.005 if gyre else 0.25, record=record,
                                   ftle=what == "ftle", seed_stride=(4.0, 4.0, 4.0),
                                   start_time=start))
    done = {}
    while len(done) < len(ids):
        r = s.server.poll(wait_ms=1000)
        if r is not None:
            if r.status:
                raise RuntimeError("request %d: status %d" % (r.id, r.status))
            done[r.id] = r
    out = []
    for i in ids:
        r = done[i]
        out.append([r.positions, r.remaining, r.termination]
                   + ([r.vertices, r.colors, r.indices] if r.vertices is not None else [])
                   + ([r.ftle] if r.ftle is not None else []))
    return out


_RUN = {"curves": _run_curves, "round": _run_round, "device": _run_device,
        "insitu": _run_insitu, "batch": _run_batch, "ftle": _run_ftle,
        "ftle_field": _run_ftle_field, "pathlines": _run_pathlines, "serve": _run_serve}


# What a pass cannot do without ------------------------------------------------


def work(case):
    """Bytes: the field once, particle state in and out, curves or FTLE out.
    Floating-point operations: 100 for a step's sample and update (four times
    that for four samples), 200 for the two samples of a time-varying field.
    Particles that leave the domain early are allowed for by counting half of
    all the iterations asked for."""
    kind = case["kind"]
    nodes = case["n0"] * case["n1"] * case["n2"]
    node = {"f32": 12, "f32_edges": 12, "f16": 6, "bf16": 6}[case.get("storage", "f32")]
    per_step = 400 if case.get("integrator") == "runge_kutta_4_true" else 100
    state = 12 + 8 + 12 + 8 + 1
    if kind == "ftle_field":
        cells = int(np.prod([n // case["stride"] for n in _shape(case)]))
        return {"bytes": cells * (12 + 4), "flops": cells * 150}
    if kind == "ftle":
        cells = int(np.prod([n // case["stride"] for n in _shape(case)]))
        steps = cells * case["iterations"] // 2
        return {"bytes": nodes * node + cells * (state + 4),
                "flops": steps * per_step + cells * 150}
    if kind == "pathlines":
        steps = case["seeds"] * case["iterations"]
        return {"bytes": nodes * case["slices"] * node + case["seeds"] * (state + 8),
                "flops": steps * 2 * per_step}
    if kind == "serve":
        plan = _request_plan(case)
        steps = sum(n * i // 2 for _, n, i, _ in plan)
        curve = sum(n * i // 2 * 24 for _, n, i, record in plan if record)
        return {"bytes": sum(n for _, n, _, _ in plan) * state + curve, "flops": steps * 100}
    if kind == "batch":
        sizes, iterations = _set_plan(case)
        steps = sum(n * i // 2 for n, i in zip(sizes, iterations))
    else:
        steps = case["seeds"] * case["iterations"] // 2
    particles = sum(sizes) if kind == "batch" else case["seeds"]
    curve = steps * (12 + 4 + 8) if kind == "curves" else 0
    field = nodes * (12 + node if kind == "insitu" else node)
    return {"bytes": field + particles * state + curve, "flops": steps * per_step}


# In 64 bits -------------------------------------------------------------------


def _locate64(x, n):
    """First nodes and weights of positions in cells; inside as the grid has it."""
    inside = ((x >= 0) & (x < torch.tensor(n, device="cuda") - 1)).all(dim=1)
    cell = torch.where(inside[:, None], x.floor(), torch.zeros_like(x))
    return inside, cell.long(), x - cell


def _sample64(flat, n, cell, w, base=0):
    """Trilinear sample, components in stored order; flat is [nodes][3]."""
    out = 0.0
    for d in range(8):
        o = (d >> 2 & 1, d >> 1 & 1, d & 1)
        index = ((cell[:, 0] + o[0]) * n[1] + cell[:, 1] + o[1]) * n[2] + cell[:, 2] + o[2] + base
        weight = 1.0
        for a in range(3):
            weight = weight * (w[:, a] if o[a] else 1 - w[:, a])
        out = out + weight[:, None] * flat[index]
    return out


def _integrate64(integrator, dt, iterations, x, velocity):
    """The reference's schemes: every stepper but the four-sample one takes one
    sample a step. velocity(x, t) gives the samples and which are valid; a
    particle stops where its sample is not, or is zero."""
    x, alive = x.double(), torch.ones(x.shape[0], dtype=torch.bool, device="cuda")
    t, last = 0.0, None
    taken = torch.zeros_like(iterations)
    for i in range(int(iterations.max())):
        v, ok = velocity(x, t)
        ok = ok & alive & (taken < iterations) & (v.abs() > 1e-5).any(dim=1)
        if integrator == "runge_kutta_4_true":
            k2, a = velocity(x + 0.5 * dt * v, t + 0.5 * dt)
            k3, b = velocity(x + 0.5 * dt * k2, t + 0.5 * dt)
            k4, c = velocity(x + dt * k3, t + dt)
            ok, move = ok & a & b & c, (v + 2 * k2 + 2 * k3 + k4) / 6
        elif integrator == "runge_kutta_dormand_prince_5" and last is not None:
            move = v + (35.0 / 384.0) * (last - v)
        else:
            move = v
        x = torch.where(ok[:, None], x + dt * move, x)
        alive, last, t = ok, v, t + dt
        taken = taken + ok
        if i % 32 == 31 and not bool(alive.any()):
            break
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "ftle_field":
        return _exact_ftle_field(case, seed) if case["mapping"] == "lattice" else None
    if kind in ("serve", "batch", "ftle"):
        return None
    n, dt = _shape(case), float(np.float32(case["step"]))
    if kind == "pathlines":
        gyre = _gyre(n, case["slices"])
        flat = torch.from_numpy(gyre.data).cuda().double().reshape(-1, 3)
        h = torch.tensor(gyre.spacing.astype(np.float64), device="cuda")
        pos, times = _pathline_starts(case["seeds"], seed)
        x, t0 = torch.from_numpy(pos).cuda(), torch.from_numpy(times).cuda().double()
        nodes = n[0] * n[1] * n[2]

        def velocity(x, t):
            inside, cell, w = _locate64(x / h, n)
            q = (t0 + t) / gyre.time_spacing
            inside = inside & (q < case["slices"] - 1)
            k = torch.where(inside, q.floor(), torch.zeros_like(q))
            u = (q - k)[:, None]
            base = k.long() * nodes
            v = (1 - u) * _sample64(flat, n, cell, w, base) \
                + u * _sample64(flat, n, cell, w, base + nodes)
            return v.flip(1), inside
    else:
        if case["iterations"] * dt / case["h"] > 120 and case["field"] == "curl":
            return None  # chaotic by then: no one position is the right one
        flat = _data(case, seed).double().reshape(-1, 3)
        h = float(np.float32(case["h"]))
        x = _seeds(case, seed, case["seeds"])

        def velocity(x, t):
            inside, cell, w = _locate64(x / h, n)
            return _sample64(flat, n, cell, w).flip(1), inside

    iterations = torch.full((x.shape[0],), case["iterations"], device="cuda")
    end = _integrate64(case["integrator"], dt, iterations, x, velocity)
    return {"position": end.cpu()}


def _exact_ftle_field(case, seed):
    _, final = _flow_map(case, seed)
    f = final.double().cpu().numpy()
    h = float(np.float32(case["h"])) * case["stride"]
    J = np.empty(f.shape + (3,))
    for d in range(3):
        index = np.arange(f.shape[d])
        after = np.take(f, np.minimum(index + 1, f.shape[d] - 1), axis=d)
        J[..., d] = (after - np.take(f, np.maximum(index - 1, 0), axis=d)) / (2 * h)
    top = np.linalg.eigvalsh(np.einsum("...ki,...kj->...ij", J, J))[..., 2]
    return np.log(np.sqrt(top)) / abs(float(np.float32(case["step"])) * case["iterations"])
