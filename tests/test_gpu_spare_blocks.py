"""Fields made and destroyed in turn, of the same, nearly the same and other sizes:
each holds its own values whatever block it was given, and reports its own size.
Calls still running on another stream when a field goes read what they were given."""
import ctypes as C

import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles
from dpa_b200 import _native as N
from bitwise import assert_same

pytestmark = pytest.mark.gpu


def _grid(shape, seed):
    rng = np.random.default_rng(seed)
    return dpa_b200.RegularGrid.from_data(rng.standard_normal(shape + (3,)), (1.0, 1.0, 1.0))


@pytest.mark.parametrize("storage", ["f32", "f16", "f32_edges"])
def test_fields_in_turn(ctx, oracle, storage):
    rng = np.random.default_rng(1)
    pos = (rng.random((500, 3)) * 18).astype(np.float32)
    rem = np.full(500, 60, np.uint64)
    sizes = [(20, 20, 20), (20, 20, 20), (20, 20, 19), (21, 20, 20), (40, 33, 20), (20, 20, 20)]
    for seed, shape in enumerate(sizes):
        grid = _grid(shape, seed)
        data = grid.data.astype(np.float16).astype(np.float32) if storage == "f16" else grid.data
        want = oracle.advect_round(oracle.OracleGrid(data, grid.spacing, grid.offset),
                                   "runge_kutta_4", 0.25, pos, rem)
        field = ctx.field(grid, storage)
        node = {"f32": 16, "f16": 8, "f32_edges": 32}[storage]
        assert field.device_bytes == int(np.prod(shape)) * node
        got = ParticleAdvector(ctx, 500, "none", "runge_kutta_4", 0.25, False, False).advect(
            field, Particles.create(pos, rem)).inactive_particles
        field.close()
        assert_same(got.position, want.positions)
        assert_same(got.termination, want.termination)


def test_a_field_destroyed_while_another_stream_reads_it(ctx, oracle):
    import torch
    grids = [_grid((64, 64, 64), s) for s in (7, 8)]
    n = 200000
    pos = (np.random.default_rng(2).random((n, 3)) * 60).astype(np.float32)
    p = torch.from_numpy(pos).cuda()
    r = torch.full((n,), 1500, dtype=torch.int64, device="cuda")
    t = torch.empty(n, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    opts = N.AdvectOptions(N.INTEGRATORS["runge_kutta_4"], 0.01, 0, 0, 0, 1, 0)
    field = ctx.field(grids[0])
    ctx.check(ctx._lib.dpa_advect_device(ctx.handle, field.handle, C.byref(opts), n,
                                         C.c_void_p(p.data_ptr()), C.c_void_p(r.data_ptr()),
                                         C.c_void_p(t.data_ptr()),
                                         C.c_void_p(stream.cuda_stream)))
    field.close()
    other = ctx.field(grids[1])  # may take the block of the first
    torch.cuda.synchronize()
    other.close()
    some = np.arange(0, n, 97)
    want = oracle.advect_round(oracle.OracleGrid(grids[0].data, grids[0].spacing, grids[0].offset),
                               "runge_kutta_4", float(np.float32(0.01)), pos[some],
                               np.full(len(some), 1500, np.uint64))
    assert_same(p.cpu().numpy()[some], want.positions)
    assert_same(t.cpu().numpy()[some], want.termination)
