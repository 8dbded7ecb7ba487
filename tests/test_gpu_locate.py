"""Locating positions by the reciprocal pair at the values its single test of
the dividends divides between the two paths: starts on the grid's lower faces
(dividends of +0 and -0), at and around 2^-64 above them, on cell boundaries and
one float beside them, and outside. Spacings inside, at the edge of and beyond
the range that the reciprocal is used for. Bit-exact with the oracle."""
import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles
from bitwise import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16", "f32_edges"])
@pytest.mark.parametrize("spacing", [0.7, 1.0 / 3.0, 3e-12, 3e-13, 7e11, 3e12])
def test_starts_on_faces_and_cell_boundaries(ctx, oracle, spacing, storage):
    rng = np.random.default_rng(5)
    data = rng.integers(-8, 9, (6, 5, 7, 3)).astype(np.float32)  # exact in 16 bits
    h = np.float32(spacing)
    grid = dpa_b200.RegularGrid.from_data(data, (h, h, h), (0.0, 0.0, 0.0))
    edge = np.array([0.0, -0.0, 2.0 ** -64, np.nextafter(np.float32(2.0 ** -64), np.float32(0)),
                     1e-45, 1e-30], np.float32)
    cells = (h * np.arange(8, dtype=np.float32)).astype(np.float32)
    beside = [np.nextafter(cells, np.float32(s)).astype(np.float32) for s in (-1.0, np.inf)]
    values = np.concatenate([edge, -edge[2:], cells, *beside, h * np.float32([0.3, 2.7])])
    pos = values[rng.integers(0, len(values), (4000, 3))].astype(np.float32)
    step = float(np.float32(0.01) * h)
    rem = np.full(pos.shape[0], 40, np.uint64)
    want = oracle.advect_round(oracle.OracleGrid(grid.data, grid.spacing, grid.offset),
                               "runge_kutta_4", step, pos, rem)
    field = ctx.field(grid, storage)
    got = ParticleAdvector(ctx, len(pos), "none", "runge_kutta_4", step, False,
                           False).advect(field, Particles.create(pos, rem)).inactive_particles
    field.close()
    assert_same(got.termination, want.termination)
    assert_same(got.remaining_iterations, want.remaining)
    assert_same(got.position, want.positions)


@pytest.mark.parametrize("spacing", [0.7, 1.0 / 3.0, 3e-13, 3e12])
def test_starts_on_slice_boundaries(ctx, oracle, spacing):
    """The time axis likewise: starts at the first slice, before it, on and
    beside later ones and past the last."""
    rng = np.random.default_rng(6)
    data = rng.integers(-8, 9, (5, 4, 6, 5, 3)).astype(np.float32)
    dt = np.float32(spacing)
    grid = dpa_b200.UnsteadyGrid.from_data(data, (0.7, 0.7, 0.7), dt)
    slices = (dt * np.arange(6, dtype=np.float32)).astype(np.float32)
    values = np.concatenate([np.float32([0.0, -0.0, 2.0 ** -64, 1e-30, -1e-30]), slices,
                             np.nextafter(slices, np.float32(-1)),
                             np.nextafter(slices, np.float32(np.inf)), dt * np.float32([0.4, 2.6])])
    pos = (rng.random((3000, 3)) * [2.1, 3.5, 2.8]).astype(np.float32)
    t0 = values[rng.integers(0, len(values), 3000)].astype(np.float32)
    step, rem = float(np.float32(0.01) * dt), np.full(3000, 30, np.uint64)
    field = ctx.field(grid)
    for integrator in ("runge_kutta_4", "runge_kutta_4_true"):
        want = oracle.advect_pathlines(grid, integrator, step, pos, t0, rem)
        got = dpa_b200.advect_pathlines(ctx, field, pos, t0, 30, integrator, step)
        assert_same(got.termination, want.termination)
        assert_same(got.position, want.positions)
        assert_same(got.time, want.times)
    field.close()
