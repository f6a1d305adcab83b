"""What one call leaves for the next: failures of asynchronous steps survive a
derivative call in between, and a wait that gave up does not fail later calls."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(vt, nx=8, ny=8, p=2, io=4):
    pb = vt.Problem(vt.make_params(nx, ny, p=p, integration_order=io, perturb_grid=0.2), vt.vortex(epsilon=0.3))
    b = vt.Batch([pb])
    dt = 0.3 * 10.0 / max(nx, ny) / ((2 * p + 1) * 17.0)
    b.set_dt([dt])
    return vt.Solver(pb), b, pb, dt


def give_up(vt, s, step):
    assert vt.lib().vt_test_bulk_wait(s._h, 200, 1) == 0
    try:
        step()
    finally:
        assert vt.lib().vt_test_bulk_wait(s._h, 0, 0) == 0


@pytest.mark.parametrize("between", ["rhs", "rhs_vjp", "rhs_jvp", "totals", "adjoint"])
def test_steps_after_a_wait_that_gave_up(vt, between):
    s, b, pb, dt = make(vt)
    U = pb.array("U0")
    s.rk4(dt, 1)
    b.rk4(1)

    def step():
        with pytest.raises(vt.VortexError) as e:
            s.rk4(dt, 3)
        assert e.value.status == vt.VT_ERR_CUDA
    give_up(vt, s, step)
    if between == "rhs":
        s.rhs()
    elif between == "totals":
        s.totals()
    elif between == "adjoint":
        s.adjoint_forward(dt, 2, 2)
        b.rk4(2)
    else:
        getattr(s, between)(U, np.ones_like(U))
    s.rk4(dt, 3)
    b.rk4(3)
    np.testing.assert_array_equal(s.download(), b.download(0))
    s.close()
    b.close()


def test_steps_after_an_unseen_wait_that_gave_up(vt):
    """rhs clears the failure of the steps that it is called on top of; the next
    steps must not rely on those all the same."""
    s, b, pb, dt = make(vt)
    give_up(vt, s, lambda: s.rk4_async(dt, 3))
    s.rhs()
    s.synchronize()
    s.rk4(dt, 3)
    b.rk4(3)
    np.testing.assert_array_equal(s.download(), b.download(0))
    s.close()
    b.close()


@pytest.mark.parametrize("nx,ny", [(8, 8), (72, 70)])
def test_jvp_keeps_the_failure_of_asynchronous_steps(vt, nx, ny):
    s, b, pb, dt = make(vt, nx, ny)
    good = pb.array("U0")
    V = np.random.default_rng(0).standard_normal(good.shape)
    want = s.rhs_jvp(good, V)
    U = good.copy()
    U[17, :, 0] = -1.0
    s.upload(U)
    s.rk4_async(dt, 2)
    np.testing.assert_array_equal(s.rhs_jvp(good, V), want)
    with pytest.raises(vt.NonPhysicalState) as e:
        s.synchronize()
    info = vt.vt_error_info()
    s.rhs_jvp(good, V)  # and the record of it
    assert vt.lib().vt_last_error(s._h, ctypes.byref(info)) == 0
    assert info.code == e.value.code != 0 and info.element == e.value.element
    s.close()
    b.close()
