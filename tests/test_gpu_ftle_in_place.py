"""FTLE written over the final positions that it is formed of, from their first value
on, from the middle and from before them, equals FTLE written elsewhere."""
import ctypes as C

import numpy as np
import pytest

import dpa_b200
from dpa_b200 import _native as N
from bitwise import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mapping", ["reference", "lattice"])
def test_ftle_over_the_final_positions(ctx, mapping):
    import torch
    shape = (67, 65, 63)
    cells = int(np.prod(shape))
    rng = np.random.default_rng(0)
    grid = dpa_b200.RegularGrid.from_data(np.zeros(shape + (3,), np.float32), (1.0, 1.0, 1.0))
    field = ctx.field(grid)
    i = np.stack(np.meshgrid(*map(np.arange, shape), indexing="ij"), -1).reshape(-1, 3)
    x = torch.from_numpy(i.astype(np.float32)).cuda()
    final = torch.from_numpy((i + rng.standard_normal(i.shape)).astype(np.float32)).cuda()
    room = torch.empty(4 * cells, device="cuda")  # one value a cell before the positions

    def run(ftle, positions):
        room[cells:] = final.reshape(-1)
        torch.cuda.synchronize()
        ctx.check(ctx._lib.dpa_ftle_estimate_device(
            ctx.handle, field.handle, (C.c_float * 3)(1, 1, 1), 50, 0.1, cells,
            C.c_void_p(x.data_ptr()), C.c_void_p(positions.data_ptr()), N.FTLE_MAPPING[mapping],
            C.c_void_p(ftle.data_ptr()), (C.c_uint64 * 3)(), None))
        ctx.synchronize()
        return ftle.cpu().numpy()

    want = run(torch.empty(cells, device="cuda"), final)
    assert np.isfinite(want).all()
    for first in (cells, 2 * cells + 17, 1, 3 * cells):
        assert_same(run(room[first:first + cells], room[cells:]), want)
    field.close()
