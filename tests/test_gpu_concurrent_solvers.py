"""Several small problems with steps under way at once: as many as have an SM for
each of their tiles take the resident kernel, the others a launch per stage.
Every one of them makes the steps that it makes alone, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def problems(vt, n):
    out = []
    for i in range(n):
        nx, ny, p = ((40, 40, 2), (64, 62, 1), (8, 8, 3), (30, 20, 2))[i % 4]
        pb = vt.Problem(vt.make_params(nx, ny, p=p, integration_order=2 * p + 2, perturb_grid=0.2),
                        vt.vortex(epsilon=0.2 + 0.01 * i))
        out.append((pb, 0.3 * 10.0 / max(nx, ny) / ((2 * p + 1) * 17.0)))
    return out


def alone(vt, pb, dt, n):
    s = vt.Solver(pb)
    for _ in range(n[1]):
        s.rk4(dt, n[0])
    U = s.download()
    s.close()
    return U


@pytest.mark.parametrize("n", [(3, 4), (12, 2), (21, 1)])
def test_threads(vt, n):
    pbs = problems(vt, 8)
    want = [alone(vt, pb, dt, n) for pb, dt in pbs]
    solvers = [vt.Solver(pb) for pb, _ in pbs]

    def steps(s, dt):
        for _ in range(n[1]):
            s.rk4(dt, n[0])

    threads = [threading.Thread(target=steps, args=(s, dt)) for s, (_, dt) in zip(solvers, pbs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, U in zip(solvers, want):
        np.testing.assert_array_equal(s.download(), U)
        s.close()


def test_asynchronous_steps_of_one_thread(vt):
    """Also with a context that is destroyed with steps under way and one that
    fails; afterwards everything is as before."""
    pbs = problems(vt, 7)
    solvers = [vt.Solver(pb) for pb, _ in pbs]
    lost, failing = vt.Solver(pbs[1][0]), vt.Solver(pbs[0][0])
    U = pbs[0][0].array("U0")
    U[3, :, 0] = -1.0
    for n in (2, 11):
        failing.upload(U)
        failing.rk4_async(pbs[0][1], 2)
        if lost is not None:
            lost.rk4_async(pbs[1][1], 3)
        for s, (_, dt) in zip(solvers, pbs):
            s.rk4_async(dt, n)
        for s in solvers:
            s.synchronize()
        with pytest.raises(vt.NonPhysicalState):
            failing.synchronize()
        if lost is not None:
            lost.close()
            lost = None
    for s, (pb, dt) in zip(solvers, pbs):
        t = vt.Solver(pb)
        t.rk4(dt, 2)
        t.rk4(dt, 11)
        np.testing.assert_array_equal(s.download(), t.download())
        t.close()
        s.close()
    failing.close()


def test_euler_steps(vt):
    (pb, dt), (other, odt) = problems(vt, 2)
    s, busy = vt.Solver(pb), vt.Solver(other)
    want = vt.Solver(pb)
    for n in (1, 4, 3):
        want.forward_euler(0.01 * dt, n)
        busy.rk4_async(odt, 5)
        s.forward_euler(0.01 * dt, n)
        busy.synchronize()
        np.testing.assert_array_equal(s.download(), want.download())
    for x in (s, busy, want):
        x.close()
