"""Small problems step in one launch (the resident kernel), larger ones and
batches by a launch per stage. Both run the same functions in the same order,
so a problem alone and the same problem as a batch of one agree bit for bit,
failures included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pair(vt, nx, ny, p, io, perturb=0.2, **kw):
    pb = vt.Problem(vt.make_params(nx, ny, p=p, integration_order=io, perturb_grid=perturb), vt.vortex(**kw))
    return vt.Solver(pb), vt.Batch([pb]), pb


def small_dt(nx, ny, p):
    return 0.3 * 10.0 / max(nx, ny) / ((2 * p + 1) * 17.0)


# one tile; ragged tiles; a single column of cells (a tile with more leaving
# faces than slots); 148 and more tiles (the largest resident grid of a B200,
# and the first that is not); every order and odd and even point counts
@pytest.mark.parametrize("nx,ny,p,io", [(4, 2, 3, 10), (5, 7, 2, 4), (27, 18, 1, 4), (1, 70, 3, 8), (8, 8, 3, 19),
                                        (64, 64, 2, 10), (32, 148, 1, 2), (32, 152, 1, 2), (9, 6, 0, 2)])
def test_steps_alone_and_in_a_batch_agree(vt, nx, ny, p, io):
    s, b, pb = pair(vt, nx, ny, p, io)
    dt = small_dt(nx, ny, p)
    b.set_dt([dt])
    for n in (1, 6):
        s.rk4(dt, n)
        b.rk4(n)
        np.testing.assert_array_equal(s.download(), b.download(0))
    s.close()
    b.close()


def test_more_steps_than_a_launch_takes(vt):
    s, b, _ = pair(vt, 8, 8, 1, 4, perturb=0.0)
    dt = small_dt(8, 8, 1)
    b.set_dt([dt])
    s.rk4(dt, 1100)
    b.rk4(1100)
    np.testing.assert_array_equal(s.download(), b.download(0))
    s.rk4(dt, 2)  # the flags go on from where the last launch left them
    b.rk4(2)
    np.testing.assert_array_equal(s.download(), b.download(0))
    s.close()
    b.close()


@pytest.mark.parametrize("n", [1, 2, 5])
def test_euler_steps(vt, n):
    """U + dt R, R from the per-stage kernel: one rounding of the product and one
    of the sum where the kernel's multiply-add has one, per step."""
    s, b, pb = pair(vt, 12, 10, 2, 6)
    dt = 0.01 * small_dt(12, 10, 2)
    U = s.download()
    want = U.copy()
    for _ in range(n):
        s.upload(want)
        want = want + dt * s.rhs()
    s.upload(U)
    s.forward_euler(dt, n)
    assert np.abs(s.download() - want).max() <= 4 * n * 1.2e-16 * np.abs(want).max()
    s.close()
    b.close()


def test_failures_are_reported_alike(vt):
    s, b, pb = pair(vt, 16, 12, 3, 6)
    dt = 40 * small_dt(16, 12, 3)  # far above the stable step: fails after some steps
    b.set_dt([dt])
    with pytest.raises(vt.NonPhysicalState) as es:
        s.rk4(dt, 50)
    with pytest.raises(vt.NonPhysicalState) as eb:
        b.rk4(50)
    for k in ("code", "element", "point", "side", "step", "stage"):
        assert getattr(es.value, k) == getattr(eb.value, k), k
    # and the context steps on as before
    U = pb.array("U0")
    s.upload(U)
    b.upload(0, U)
    ok = small_dt(16, 12, 3)
    b.set_dt([ok])
    s.rk4(ok, 3)
    b.rk4(3)
    np.testing.assert_array_equal(s.download(), b.download(0))
    s.close()
    b.close()


def test_a_wait_that_gives_up(vt):
    """No copies are issued: the resident kernel's wait runs out, the call says
    so, the state is unchanged and the context steps as before afterwards."""
    s, b, pb = pair(vt, 8, 8, 2, 4)
    U = s.download()
    dt = small_dt(8, 8, 2)
    assert vt.lib().vt_test_bulk_wait(s._h, 200, 1) == 0
    with pytest.raises(vt.VortexError) as e:
        s.rk4(dt, 2)
    assert e.value.status == vt.VT_ERR_CUDA
    np.testing.assert_array_equal(s.download(), U)
    assert vt.lib().vt_test_bulk_wait(s._h, 0, 0) == 0
    b.set_dt([dt])
    s.rk4(dt, 2)
    b.rk4(2)
    np.testing.assert_array_equal(s.download(), b.download(0))
    s.close()
    b.close()


@pytest.mark.parametrize("nx,ny,p,io", [(5, 7, 3, 10), (8, 8, 1, 3), (27, 18, 1, 4), (9, 6, 0, 2)])
def test_operators_as_they_are(vt, nx, ny, p, io):
    """The form without folded operators has half the threads and more points
    of a face side by side (2, 3 and more of them per item here)."""
    import ctypes
    s, b, pb = pair(vt, nx, ny, p, io)
    dt = small_dt(nx, ny, p)
    s.stage_mapping = 0
    assert vt.lib().vt_batch_set_mapping(b._h, (ctypes.c_int * 1)(0)) == 0
    b.set_dt([dt])
    s.rk4(dt, 5)
    b.rk4(5)
    np.testing.assert_array_equal(s.download(), b.download(0))
    s.close()
    b.close()
