"""How a recording round's curve is handed to the sink: in one chunk unless it exceeds
the limit, which a sink that appends to growing arrays depends on, else in as few as the
limit allows; the same curve either way."""
import ctypes as C

import numpy as np
import pytest

import dpa_b200
from dpa_b200 import Particles
from dpa_b200 import _native as N
from bitwise import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index64", [0, 1])
@pytest.mark.parametrize("seeds", [2000, 20000])
def test_chunks(seeds, index64):
    grid = dpa_b200.fields.abc(32)
    iterations = 1200000 // seeds
    rng = np.random.default_rng(seeds)
    start = (rng.random((seeds, 3)) * 4 + 1).astype(np.float32)
    options = N.AdvectOptions(N.INTEGRATORS["runge_kutta_4"], 0.001, 1, index64, 1, 1, 0)
    itype = np.uint64 if index64 else np.uint32
    with dpa_b200.Context(0) as ctx:
        field = ctx.field(grid)

        def run(limit):
            if limit:
                ctx.check(ctx._lib.dpa_context_set_host_chunk_limit(ctx.handle, limit))
            chunks, parts = [], []

            def take(user, chunk):
                c = chunk.contents
                v, i = int(c.vertex_count), int(c.index_count)
                chunks.append((int(c.vertex_offset), v, int(c.index_offset), i, int(c.last)))
                ptr = C.cast(c.indices, C.POINTER(C.c_uint64 if index64 else C.c_uint32))
                parts.append((np.ctypeslib.as_array(c.vertices, (v * 3,)).copy(),
                              np.ctypeslib.as_array(c.colors, (v,)).copy(),
                              np.ctypeslib.as_array(ptr, (i,)).copy() if i else
                              np.zeros(0, itype)))
                return 0
            p = Particles.create(start, iterations)
            ctx.check(ctx._lib.dpa_advect_round(
                ctx.handle, field.handle, C.byref(options), seeds,
                p.position.ctypes.data_as(C.c_void_p),
                p.remaining_iterations.ctypes.data_as(C.c_void_p), None,
                N.CURVE_SINK(take), None))
            return chunks, [np.concatenate(a) for a in zip(*parts)]

        chunks, want = run(0)
        assert len(want[1]) > 1000000
        assert chunks == [(0, len(want[1]), 0, len(want[2]), 1)]
        limit = 1 << 20
        chunks, got = run(limit)
        most_v, most_i = limit // 16, limit // itype().nbytes
        assert len(chunks) == max(-(-len(want[1]) // most_v), -(-len(want[2]) // most_i))
        assert all(c[1] <= most_v and c[3] <= most_i for c in chunks)
        assert [c[4] for c in chunks] == [0] * (len(chunks) - 1) + [1]
        for a, b in zip(got, want):
            assert_same(a, b)
        field.close()
