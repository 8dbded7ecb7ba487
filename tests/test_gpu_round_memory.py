"""The device memory that a context's first recording round takes: its raw curves and
the curve that survives, not room for every raw vertex again where most particles leave
early."""
import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles

pytestmark = pytest.mark.gpu


def test_first_recording_round(ctx):
    import torch
    ctx.set_spare_limit(0)
    data = np.zeros((16, 16, 16, 3), np.float32)
    data[..., 2] = 1.0  # along axis 0, out of the field within 60 steps
    grid = dpa_b200.RegularGrid.from_data(data, (1, 1, 1))
    n, iterations = 4096, 1000
    pos = (np.random.default_rng(0).random((n, 3)) * 15).astype(np.float32)

    def round_of(context, field, count):
        out = ParticleAdvector(context, count, "none", "runge_kutta_4", 0.25, False, True).advect(
            field, Particles.create(pos[:count], iterations))
        return len(out.integral_curves[0].vertices)

    with dpa_b200.Context(0) as first:  # loads the code
        field = first.field(grid)
        round_of(first, field, n)
        field.close()
    with dpa_b200.Context(0) as context:
        field = context.field(grid)
        round_of(context, field, 10)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        vertices = round_of(context, field, n)
        taken = before - torch.cuda.mem_get_info()[0]
        assert vertices < n * 64
        # 12 bytes a raw vertex; 24 a surviving one; the particles; 2 MiB for each of a
        # dozen arrays.
        assert taken <= n * (iterations + 2) * 12 + vertices * 24 + n * 64 + (24 << 20)
        field.close()
    ctx.set_spare_limit(1 << 30)
