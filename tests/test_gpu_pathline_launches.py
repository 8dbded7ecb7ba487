"""Pathlines at the count where a launch no longer fits the SMs at once and another
build of the kernel takes over (148 SMs of 512 threads): bit-exact with the oracle
on both sides of it, for each way to divide by the spacing, from F32 nodes and edge
records."""
import numpy as np
import pytest

import dpa_b200
from dpa_b200 import UnsteadyGrid, fields
from bitwise import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f32", "f32_edges"])
@pytest.mark.parametrize("integrator", ["runge_kutta_4", "euler"])
@pytest.mark.parametrize("spacing", [None, 0.25, 3e-13])
@pytest.mark.parametrize("count", [75776, 75777, 151553])
def test_pathlines_beyond_one_wave(ctx, oracle, count, spacing, integrator, storage):
    gyre = fields.double_gyre((16, 8, 8), 5)
    extent = np.array([2.0, 1.0, 1.0])
    step = 0.05
    if spacing is not None:
        extent = np.array([15.0, 7.0, 7.0]) * spacing
        gyre = UnsteadyGrid.from_data(gyre.data, [spacing] * 3, gyre.time_spacing)
        step = 0.4 * spacing
    rng = np.random.default_rng(count)
    pos = (rng.random((count, 3)) * extent * 1.02).astype(np.float32)  # some start outside
    times = (rng.random(count) * 10.5).astype(np.float32)
    rem = rng.integers(0, 30, count).astype(np.uint64)
    want = oracle.advect_pathlines(gyre, integrator, step, pos, times, rem)
    field = ctx.field(gyre, storage)
    got = dpa_b200.advect_pathlines(ctx, field, pos, times, rem, integrator, step)
    field.close()
    assert_same(got.termination, want.termination)
    assert_same(got.remaining_iterations, want.remaining)
    assert_same(got.position, want.positions)
    assert_same(got.time, want.times)
