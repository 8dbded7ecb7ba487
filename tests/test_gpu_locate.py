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
