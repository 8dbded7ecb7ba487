"""Launches small enough for 1, 2, 4, 8 or 16 particles per warp, at the counts
where the number changes on 148 SMs, recording and not, steady and not: bit-exact
with the oracle."""
import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles, fields
from bitwise import assert_same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grids():
    return fields.curl_noise(24, 3.0, 3), fields.double_gyre((16, 8, 8), 5)


@pytest.mark.parametrize("count", [1, 2, 1024, 1025, 1184, 1185, 2368, 2369, 4737, 9473, 18944, 18945])
def test_particles_per_warp(ctx, oracle, grids, count):
    steady, gyre = grids
    rng = np.random.default_rng(count)
    pos = (rng.random((count, 3)) * 23.5).astype(np.float32)  # some start outside
    rem = rng.integers(0, 40, count).astype(np.uint64)
    og = oracle.OracleGrid(steady.data, steady.spacing, steady.offset)
    field = ctx.field(steady)
    for record in (False, True):
        want = oracle.advect_round(og, "runge_kutta_4", 0.25, pos, rem, record=record)
        got = ParticleAdvector(ctx, count, "none", "runge_kutta_4", 0.25, False, record).advect(
            field, Particles.create(pos, rem))
        assert_same(got.inactive_particles.termination, want.termination)
        assert_same(got.inactive_particles.remaining_iterations, want.remaining)
        assert_same(got.inactive_particles.position, want.positions)
        if record:
            assert_same(got.integral_curves[0].vertices, want.vertices)
            assert_same(got.integral_curves[0].indices, want.indices)
    field.close()
    pos = (rng.random((count, 3)) * [2.0, 1.0, 1.0]).astype(np.float32)
    times = (rng.random(count) * 10.5).astype(np.float32)
    want = oracle.advect_pathlines(gyre, "runge_kutta_4", 0.05, pos, times, rem)
    field = ctx.field(gyre)
    got = dpa_b200.advect_pathlines(ctx, field, pos, times, rem, "runge_kutta_4", 0.05)
    field.close()
    assert_same(got.termination, want.termination)
    assert_same(got.position, want.positions)
    assert_same(got.time, want.times)
