"""The processing order at the sizes where its counting sort divides: one bucket,
counters that end just behind a tile of the scan, one tile and all of them; a
count with a ragged last block; starts in one bucket, anywhere and all outside.
Every particle is advected once whatever the order: bit-exact with the oracle."""
import ctypes as C

import numpy as np
import pytest

from dpa_b200 import ParticleAdvector, Particles, fields
from dpa_b200 import _native as N
from bitwise import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("starts", ["one", "any", "outside"])
@pytest.mark.parametrize("resolution,count", [(1, 8192), (8, 8193), (10, 8449), (33, 70001),
                                              (64, 8192), (64, 200003)])
def test_every_particle_is_in_the_order_once(ctx, oracle, resolution, count, starts):
    grid = fields.curl_noise(33, 4.0, 1)
    rng = np.random.default_rng(resolution + count)
    pos = (rng.random((count, 3)) * 33.0 - 0.5).astype(np.float32)  # some outside
    if starts == "one":
        pos = (4.0 + pos * 1e-3).astype(np.float32)
    elif starts == "outside":
        pos[:, rng.integers(0, 3)] = rng.choice([-1.0, 40.0, np.nan], count)
    rem = rng.integers(0, 20, count).astype(np.uint64)
    want = oracle.advect_round(oracle.OracleGrid(grid.data, grid.spacing, grid.offset),
                               "runge_kutta_4", 0.25, pos, rem)
    saved = N.Tuning()
    ctx.check(ctx._lib.dpa_context_get_tuning(ctx.handle, C.byref(saved)))
    tuning = N.Tuning()
    ctx.check(ctx._lib.dpa_context_get_tuning(ctx.handle, C.byref(tuning)))
    tuning.order = resolution
    field = ctx.field(grid)
    try:
        ctx.check(ctx._lib.dpa_context_set_tuning(ctx.handle, C.byref(tuning)))
        got = ParticleAdvector(ctx, count, "none", "runge_kutta_4", 0.25, False, False).advect(
            field, Particles.create(pos, rem)).inactive_particles
    finally:
        ctx.check(ctx._lib.dpa_context_set_tuning(ctx.handle, C.byref(saved)))
        field.close()
    assert_same(got.termination, want.termination)
    assert_same(got.remaining_iterations, want.remaining)
    assert_same(got.position, want.positions)
