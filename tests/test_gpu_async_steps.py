"""Asynchronous steps, many of which are replayed from a graph, are the
synchronous ones, bit for bit, whatever changed since the graph was made."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def small_dt(n, p):
    return 0.3 * 10.0 / n / ((2 * p + 1) * 17.0)


@pytest.mark.parametrize("nx,ny,p", [(72, 70, 2), (8, 8, 1)])
def test_asynchronous_steps(vt, nx, ny, p):
    pb = vt.Problem(vt.make_params(nx, ny, p=p, integration_order=2 * p + 2, perturb_grid=0.2), vt.vortex(epsilon=0.3))
    dt = small_dt(nx, p)
    a, s = vt.Solver(pb), vt.Solver(pb)

    def steps(n, h=dt):
        a.rk4_async(h, n)
        a.synchronize()
        s.rk4(h, n)
        np.testing.assert_array_equal(a.download(), s.download())
        assert a.time == s.time

    for n in (7, 8, 11, 30):  # below, at and beside multiples of the graph's steps
        steps(n)
    steps(9, 0.5 * dt)
    for x in (a, s):
        x.forward_euler(0.01 * dt, 1)  # the state is in the other buffer now
    steps(13, 0.5 * dt)
    for x in (a, s):
        x.stage_mapping = 0
    steps(10, 0.5 * dt)
    U = pb.array("U0")
    U[11, :, 0] = -1.0
    a.upload(U)
    a.rk4_async(0.5 * dt, 10)
    with pytest.raises(vt.NonPhysicalState) as e:
        a.synchronize()
    s.upload(U)
    with pytest.raises(vt.NonPhysicalState) as f:
        s.rk4(0.5 * dt, 10)
    assert (e.value.element, e.value.step, e.value.stage) == (f.value.element, f.value.step, f.value.stage)
    assert e.value.step == 0
    a.close()
    s.close()
