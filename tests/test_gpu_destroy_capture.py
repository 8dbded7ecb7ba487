"""A field destroyed by one thread while another captures a graph on the same device:
the capture ends as it should and replays, and neither thread's next launch fails.
Fields used in the context's stream, in another one, and in a graph."""
import ctypes as C
import threading

import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles
from dpa_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use", ["own stream", "other stream", "graph"])
def test_destroy_beside_a_capture(use):
    import torch
    rng = np.random.default_rng(0)
    grid = dpa_b200.RegularGrid.from_data(rng.standard_normal((20, 20, 20, 3)), (1.0, 1.0, 1.0))
    n = 1000
    pos = (rng.random((n, 3)) * 19).astype(np.float32)
    particles = Particles.create(pos, 20)
    p = torch.from_numpy(pos).cuda()
    r = torch.full((n,), 20, dtype=torch.int64, device="cuda")
    term = torch.empty(n, dtype=torch.uint8, device="cuda")
    side, capturing = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.ones(1000, device="cuda")
    torch.cuda.synchronize()
    opts = N.AdvectOptions(N.INTEGRATORS["runge_kutta_4"], 0.25, 0, 0, 0, 1, 0)
    ready, captures, done = (threading.Event() for _ in range(3))
    errors = []

    def destroyer():
        try:
            with dpa_b200.Context(0) as ctx:
                advector = ParticleAdvector(ctx, n, "none", "runge_kutta_4", 0.25, False, False)
                field, kept = ctx.field(grid), ctx.field(grid)
                want = advector.advect(kept, particles).inactive_particles.position
                advector.advect(field, particles)
                arrays = [C.c_void_p(a.data_ptr()) for a in (p, r, term)]
                if use == "other stream":
                    ctx.check(ctx._lib.dpa_advect_device(ctx.handle, field.handle, C.byref(opts),
                                                         n, *arrays, C.c_void_p(side.cuda_stream)))
                if use == "graph":
                    graph = C.c_void_p()
                    ctx.check(ctx._lib.dpa_graph_create_advect(
                        ctx.handle, field.handle, C.byref(opts), n, *arrays, C.byref(graph)))
                    ctx.check(ctx._lib.dpa_graph_launch(ctx.handle, graph,
                                                        C.c_void_p(side.cuda_stream)))
                    ctx.check(ctx._lib.dpa_graph_destroy(ctx.handle, graph))
                ready.set()
                assert captures.wait(60)
                status = ctx._lib.dpa_field_destroy(ctx.handle, field.handle)
                field.handle = None
                ctx.check(status)
                got = advector.advect(kept, particles).inactive_particles.position
                np.testing.assert_array_equal(got, want)
                done.set()
                kept.close()
        except Exception as e:  # for the test's own thread
            errors.append(e)
        finally:
            ready.set()
            done.set()

    thread = threading.Thread(target=destroyer)
    thread.start()
    assert ready.wait(60)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(capturing):
        graph.capture_begin(capture_error_mode="thread_local")
        x.mul_(2.0)
        captures.set()
        assert done.wait(60)
        graph.capture_end()
    thread.join()
    assert not errors, errors
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 2.0).all()
