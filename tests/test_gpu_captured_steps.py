"""A caller may capture asynchronous steps on the context's stream and replay
them: every replay makes the same steps again, also where steps that are not
captured take one launch for all of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,p", [(8, 8, 2), (64, 66, 1), (72, 70, 2)])
def test_replays(vt, nx, ny, p):
    import torch

    pb = vt.Problem(vt.make_params(nx, ny, p=p, integration_order=2 * p + 2, perturb_grid=0.2), vt.vortex(epsilon=0.3))
    dt = 0.3 * 10.0 / max(nx, ny) / ((2 * p + 1) * 17.0)
    s, b = vt.Solver(pb), vt.Batch([pb])
    b.set_dt([dt])
    s.rk4(dt, 1)
    b.rk4(1)
    stream = torch.cuda.ExternalStream(s.stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        s.rk4_async(dt, 3)
        graph.capture_end()
    s.synchronize()
    np.testing.assert_array_equal(s.download(), b.download(0))  # nothing was run yet
    for replays in (1, 2, 1):
        with torch.cuda.stream(stream):
            for _ in range(replays):
                graph.replay()
        stream.synchronize()
        b.rk4(3 * replays)
        np.testing.assert_array_equal(s.download(), b.download(0))
        s.rk4(dt, 2)  # steps that are not captured, in between
        b.rk4(2)
        np.testing.assert_array_equal(s.download(), b.download(0))
    del graph
    s.close()
    b.close()
