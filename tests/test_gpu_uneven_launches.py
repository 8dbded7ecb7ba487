"""Launches of one to four blocks per SM (148 SMs, blocks of 256), at the counts where
they are dealt out in smaller blocks and where not, steady and not, recording and not:
bit-exact with the oracle."""
import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles, fields
from bitwise import assert_same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grids():
    return fields.curl_noise(24, 3.0, 3), fields.double_gyre((16, 8, 8), 5)


@pytest.mark.parametrize("count", [37888, 37889, 60671, 60672, 75777, 90881, 113665, 121089, 151553])
def test_uneven_launches(ctx, oracle, grids, count):
    steady, gyre = grids
    rng = np.random.default_rng(count)
    pos = (rng.random((count, 3)) * 23.5).astype(np.float32)  # some start outside
    rem = rng.integers(0, 12, count).astype(np.uint64)
    og = oracle.OracleGrid(steady.data, steady.spacing, steady.offset)
    field = ctx.field(steady)
    for record, integrator in ((False, "runge_kutta_4"), (True, "runge_kutta_4"),
                               (False, "runge_kutta_4_true")):
        want = oracle.advect_round(og, integrator, 0.25, pos, rem, record=record)
        got = ParticleAdvector(ctx, count, "none", integrator, 0.25, False, record).advect(
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
