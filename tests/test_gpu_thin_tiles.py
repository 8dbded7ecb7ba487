"""Tiled fields that are thin along axis 2, or just above a tile there: at most an
eighth more memory than their rows, and no more than their rows where there is no room
for tiles. One and two particles per lane, bit-exact with the oracle."""
import ctypes as C

import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles
from dpa_b200 import _native as N
from bitwise import assert_same

pytestmark = pytest.mark.gpu

NODE_BYTES = {"f32": 16, "f16": 8}


def _check(context, oracle, grid, field):
    rng = np.random.default_rng(5)
    n, shape = 4000, np.array(grid.shape)
    pos = (rng.random((n, 3)) * (shape - 1)).astype(np.float32)
    rem = np.full(n, 25, np.uint64)
    want = oracle.advect_round(oracle.OracleGrid(grid.data, grid.spacing, grid.offset),
                               "runge_kutta_4", 0.0625, pos, rem)
    for lanes in (1, 2):
        tuning = N.Tuning(16, 0, 64, 0.0, 0, lanes)
        context.check(context._lib.dpa_context_set_tuning(context.handle, C.byref(tuning)))
        got = ParticleAdvector(context, n, "none", "runge_kutta_4", 0.0625, False, False).advect(
            field, Particles.create(pos, rem)).inactive_particles
        assert_same(got.termination, want.termination)
        assert_same(got.position, want.positions)


def _grid(shape):
    data = np.random.default_rng(7).integers(-8, 9, shape + (3,), np.int8).astype(np.float32)
    return dpa_b200.RegularGrid.from_data(data, (1, 1, 1))


@pytest.mark.parametrize("storage,shape", [
    ("f32", (4100, 4100, 2)), ("f32", (3350, 3349, 3)), ("f32", (1021, 1000, 33)),
    ("f16", (4099, 4098, 4)), ("f16", (1021, 1013, 65))])
def test_thin_tiles(oracle, storage, shape):
    grid = _grid(shape)
    with dpa_b200.Context(0) as context:
        field = context.field(grid, storage)
        rows = int(np.prod(shape)) * NODE_BYTES[storage]
        assert 512 << 20 <= rows < field.device_bytes <= rows * 9 // 8
        _check(context, oracle, grid, field)
        field.close()


def test_rows_where_tiles_find_no_room(ctx, oracle):
    import torch
    shape = (65, 15645, 33)  # the tiles take 11 % more than the rows
    grid = _grid(shape)
    rows = int(np.prod(shape)) * 16
    ctx.set_spare_limit(0)  # a failed allocation would give back what others keep
    data = torch.from_numpy(grid.data).cuda()
    with dpa_b200.Context(0) as context:
        dpa_b200.Field(context, grid, "f32", device_pointer=data.data_ptr()).close()
        context.set_spare_limit(0)
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - rows - (30 << 20), dtype=torch.uint8,
                           device="cuda")
        assert rows <= torch.cuda.mem_get_info()[0] <= rows + (40 << 20)
        field = dpa_b200.Field(context, grid, "f32", device_pointer=data.data_ptr())
        assert field.device_bytes == rows
        _check(context, oracle, grid, field)
        field.close()
        del fill, data
        torch.cuda.empty_cache()
    ctx.set_spare_limit(1 << 30)
