"""Tunings that limit the blocks per SM and leave the block size to the launch, at
counts around one and two blocks of 256 per SM (148 SMs), one and two particles per
lane: bit-exact with the oracle."""
import ctypes as C

import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles, fields
from dpa_b200 import _native as N
from bitwise import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [37889, 50000, 75777])
@pytest.mark.parametrize("blocks_per_sm,lanes", [(1, 1), (2, 1), (4, 1), (1, 2)])
def test_blocks_per_sm(oracle, count, blocks_per_sm, lanes):
    grid = fields.curl_noise(24, 3.0, 3)
    rng = np.random.default_rng(count)
    pos = (rng.random((count, 3)) * 23.5).astype(np.float32)  # some start outside
    rem = rng.integers(0, 12, count).astype(np.uint64)
    want = oracle.advect_round(oracle.OracleGrid(grid.data, grid.spacing, grid.offset),
                               "runge_kutta_4", 0.25, pos, rem)
    with dpa_b200.Context(0) as ctx:
        tuning = N.Tuning(16, blocks_per_sm, 64, 0.0, 0, lanes)
        ctx.check(ctx._lib.dpa_context_set_tuning(ctx.handle, C.byref(tuning)))
        field = ctx.field(grid)
        got = ParticleAdvector(ctx, count, "none", "runge_kutta_4", 0.25, False, False).advect(
            field, Particles.create(pos, rem)).inactive_particles
        field.close()
    assert_same(got.termination, want.termination)
    assert_same(got.remaining_iterations, want.remaining)
    assert_same(got.position, want.positions)
