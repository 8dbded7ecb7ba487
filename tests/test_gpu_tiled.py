"""Fields large enough to be laid out in tiles: starts beside tile borders, at the
grid's faces and anywhere, bit-exact with the oracle. Axes are no multiples of the
tile sizes, one is a single cell, one spacing is no power of two."""
import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles
from bitwise import assert_same

pytestmark = pytest.mark.gpu

NODE_BYTES = {"f32": 16, "f16": 8, "bf16": 8, "f32_edges": 32}


@pytest.mark.parametrize("storage,shape,spacing", [
    ("f32", (323, 322, 325), 1.0), ("f32", (2, 4100, 4100), 0.7),
    ("f16", (406, 407, 411), 0.7), ("bf16", (3, 5, 4500001), 1.0),
    ("f32_edges", (257, 259, 254), 0.7), ("f32_edges", (4200, 4100, 2), 1.0)])
def test_tiled_fields_match_the_oracle(ctx, oracle, storage, shape, spacing):
    rng = np.random.default_rng(7)
    data = rng.integers(-8, 9, shape + (3,), np.int8).astype(np.float32)  # exact in 16 bits
    h = np.float32(spacing)
    grid = dpa_b200.RegularGrid.from_data(data, (h, h, h))
    field = ctx.field(grid, storage)
    # More than the rows alone would take: the field is tiled.
    assert field.device_bytes > np.prod(shape) * NODE_BYTES[storage] >= 512 << 20
    n, want = 3000, (64, 32 if storage == "f32_edges" else 64,
                     32 if storage.startswith("f32") else 64)
    cell = np.empty((n, 3))
    for axis, size in enumerate(shape):
        tiles = -(-size // want[axis])
        tile = -(-size // tiles)
        border = rng.integers(0, tiles + 1, n) * tile + rng.integers(-2, 2, n)
        anywhere = rng.integers(0, size, n)
        at = np.where(rng.random(n) < 0.7, border, anywhere)
        cell[:, axis] = np.clip(at, 0, size - 2) + rng.random(n)
    pos = (cell.astype(np.float32) * h).astype(np.float32)
    rem, step = np.full(n, 25, np.uint64), float(np.float32(0.06) * h)
    og = oracle.OracleGrid(grid.data, grid.spacing, grid.offset)
    for integrator, record in (("runge_kutta_4", False), ("runge_kutta_4_true", False),
                               ("runge_kutta_4", True)):
        want_ = oracle.advect_round(og, integrator, step, pos, rem, record=record)
        got = ParticleAdvector(ctx, n, "none", integrator, step, False, record).advect(
            field, Particles.create(pos, rem))
        assert_same(got.inactive_particles.termination, want_.termination)
        assert_same(got.inactive_particles.remaining_iterations, want_.remaining)
        assert_same(got.inactive_particles.position, want_.positions)
        if record:
            assert_same(got.integral_curves[0].vertices, want_.vertices)
            assert_same(got.integral_curves[0].indices, want_.indices)
    field.close()
