"""A graph destroyed by one thread, right behind a replay in another stream, while another
thread captures on the same device: the capture ends as it should and replays, the
destroyed graph's last replay finishes, and the thread's next launch does not fail."""
import ctypes as C
import threading

import numpy as np
import pytest

import dpa_b200
from dpa_b200 import ParticleAdvector, Particles
from dpa_b200 import _native as N

pytestmark = pytest.mark.gpu


# Below and above the fewest particles that are ordered first.
@pytest.mark.parametrize("n", [1000, 20000])
def test_graph_destroyed_beside_a_capture(n):
    import torch
    rng = np.random.default_rng(0)
    grid = dpa_b200.RegularGrid.from_data(rng.standard_normal((20, 20, 20, 3)), (1.0, 1.0, 1.0))
    pos = (rng.random((n, 3)) * 19).astype(np.float32)
    p = torch.from_numpy(pos).cuda()
    r = torch.full((n,), 20, dtype=torch.int64, device="cuda")
    term = torch.empty(n, dtype=torch.uint8, device="cuda")
    side, capturing = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.ones(1000, device="cuda")
    torch.cuda.synchronize()
    opts = N.AdvectOptions(N.INTEGRATORS["runge_kutta_4"], 0.25, 0, 0, 0, 1, 0)
    ready, captures, done = (threading.Event() for _ in range(3))
    errors, wants = [], []

    def destroyer():
        try:
            with dpa_b200.Context(0) as ctx:
                advector = ParticleAdvector(ctx, n, "none", "runge_kutta_4", 0.25, False, False)
                field = ctx.field(grid)
                particles = Particles.create(pos, 20)
                wants.append(advector.advect(field, particles).inactive_particles.position)
                graph = C.c_void_p()
                arrays = [C.c_void_p(a.data_ptr()) for a in (p, r, term)]
                ctx.check(ctx._lib.dpa_graph_create_advect(
                    ctx.handle, field.handle, C.byref(opts), n, *arrays, C.byref(graph)))
                ready.set()
                assert captures.wait(60)
                ctx.check(ctx._lib.dpa_graph_launch(ctx.handle, graph,
                                                    C.c_void_p(side.cuda_stream)))
                ctx.check(ctx._lib.dpa_graph_destroy(ctx.handle, graph))
                got = advector.advect(field, particles).inactive_particles.position
                np.testing.assert_array_equal(got, wants[0])
                done.set()
                field.close()
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
    np.testing.assert_array_equal(p.cpu().numpy(), wants[0])
