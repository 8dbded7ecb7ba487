"""Fields whose limit of threads per SM depends on the length of a launch's steps: short
and long ones, more particles than fit at once, bit-exact with the oracle."""
import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles
from bitwise import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,shape", [("f32_edges", (350, 349, 353)),
                                           ("f16", (551, 553, 557))])
def test_short_and_long_steps(ctx, oracle, storage, shape):
    rng = np.random.default_rng(3)
    data = rng.integers(-8, 9, shape + (3,), np.int8).astype(np.float32)  # exact in 16 bits
    data[rng.random(shape) < 1e-4] = np.inf  # not part of the speed that the limit goes by
    grid = dpa_b200.RegularGrid.from_data(data, (1.0, 0.5, 1.0))
    og = oracle.OracleGrid(grid.data, grid.spacing, grid.offset)
    field = ctx.field(grid, storage)
    assert 1280 << 20 < field.device_bytes <= 3 << 30
    n = 200000
    pos = (rng.random((n, 3)) * (np.array(shape) - 1) * [1, 0.5, 1]).astype(np.float32)
    rem = rng.integers(0, 12, n).astype(np.uint64)
    for step in (0.01, -0.0625):  # 0.1 and 0.6 cells along an axis
        want = oracle.advect_round(og, "runge_kutta_4", step, pos, rem)
        got = ParticleAdvector(ctx, n, "none", "runge_kutta_4", step, False, False).advect(
            field, Particles.create(pos, rem)).inactive_particles
        assert_same(got.termination, want.termination)
        assert_same(got.remaining_iterations, want.remaining)
        assert_same(got.position, want.positions)
    field.close()
