"""Recording rounds around the particle count up to which one block scans the curve
offsets: two launches fewer up to there, and the curve bit-exact with the oracle on both
sides."""
import ctypes as C

import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles, fields
from bitwise import assert_same

pytestmark = pytest.mark.gpu


def _launches(ctx):
    n = C.c_uint64()
    ctx.check(ctx._lib.dpa_context_launch_count(ctx.handle, C.byref(n)))
    return n.value


def test_curve_offsets_around_one_block(oracle):
    grid = fields.curl_noise(24, 3.0, 3)
    og = oracle.OracleGrid(grid.data, grid.spacing, grid.offset)
    launches = {}
    with dpa_b200.Context(0) as ctx:
        field = ctx.field(grid)
        for count in (3071, 3072, 3073, 4096, 5000):
            rng = np.random.default_rng(count)
            pos = (rng.random((count, 3)) * 23.5).astype(np.float32)  # some start outside
            rem = rng.integers(0, 40, count).astype(np.uint64)
            want = oracle.advect_round(og, "runge_kutta_4", 0.25, pos, rem, record=True)
            before = _launches(ctx)
            got = ParticleAdvector(ctx, count, "none", "runge_kutta_4", 0.25, False,
                                   True).advect(field, Particles.create(pos, rem))
            launches[count] = _launches(ctx) - before
            assert_same(got.integral_curves[0].vertices, want.vertices)
            assert_same(got.integral_curves[0].indices, want.indices)
        field.close()
    assert launches[3071] == launches[3072]
    assert launches[3073] == launches[4096] == launches[5000] == launches[3072] + 2
