"""What a context keeps of destroyed fields: nothing of a program that makes one field,
the blocks of a program that makes many, no more than the limit, and a field too large
to be kept takes no other's place."""
import numpy as np
import pytest

import dpa_b200

pytestmark = pytest.mark.gpu

SLACK = 8 << 20  # allocation granularity, and what the driver keeps for itself


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _grid(n):
    return dpa_b200.RegularGrid.from_data(np.zeros((n, 160, 160, 3), np.float32), (1, 1, 1))


@pytest.fixture
def own(ctx):
    ctx.set_spare_limit(0)  # a failed allocation would give back what others keep
    with dpa_b200.Context(0) as context:
        context.field(_grid(160)).close()  # loads the code
        context.set_spare_limit(0)
        context.set_spare_limit(1 << 30)
        yield context
    ctx.set_spare_limit(1 << 30)


def test_one_field_keeps_no_upload_copy(own):
    before = _free()
    field = own.field(_grid(200))
    nodes = 200 * 160 * 160
    assert nodes * 16 - SLACK <= before - _free() <= nodes * 16 + SLACK
    field.close()
    assert nodes * 16 - SLACK <= before - _free() <= nodes * 16 + SLACK
    own.field(_grid(200)).close()  # of the kept block: its copy is kept as well
    assert nodes * 28 - SLACK <= before - _free() <= nodes * 28 + SLACK
    own.set_spare_limit(nodes * 28 - 1)  # the older one goes
    assert nodes * 12 - SLACK <= before - _free() <= nodes * 16 + SLACK
    own.set_spare_limit(0)
    assert abs(before - _free()) <= SLACK
    own.field(_grid(200)).close()
    assert abs(before - _free()) <= SLACK


def test_a_field_above_the_limit_takes_no_place(own):
    before = _free()
    own.field(_grid(200)).close()
    kept = before - _free()
    assert kept >= 200 * 160 * 160 * 16 - SLACK
    own.field(_grid(2700)).close()  # 1.03 GiB
    assert abs(before - _free() - kept) <= SLACK


def test_no_more_than_four_blocks(own):
    before = _free()
    for n in (100, 150, 225, 340, 510, 770):
        own.field(_grid(n)).close()
    held = (225 + 340 + 510 + 770) * 160 * 160 * 16
    assert held - SLACK <= before - _free() <= held + SLACK
