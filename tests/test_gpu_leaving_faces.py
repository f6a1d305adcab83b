"""Tiles with more leaving faces than the 24 slots per half: three columns of
cells (31 and 32 per half), and the structured mesh with its elements in another
order (any mesh but the reference's own comes in tiles of 64 consecutive
elements: up to 96 per half). Every kernel has a form for them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def small_dt(nx, ny, p):
    return 0.3 * 10.0 / max(nx, ny) / ((2 * p + 1) * 17.0)


class Reordered:
    """A structured problem with element perm[i] as its element i."""

    def __init__(self, vt, pb, perm, stiff=None):
        inv = np.empty_like(perm)
        inv[perm] = np.arange(len(perm))
        self.K, self.Np, self.p, self.perm = pb.K, pb.Np, pb.p, perm
        self.U = pb.array("U0")[perm]
        self.desc, self.keep = vt.mesh_desc_from_arrays(
            pb.p, pb.array("type")[perm], inv[pb.array("conn")[perm]], pb.array("detj")[perm], pb.array("jinv")[perm],
            pb.array("normals")[perm], pb.array("sides")[perm], pb.array("minv_ref"),
            pb.array("stiff_ref") if stiff is None else stiff, pb.array("line_quad"), pb.array("phi_plus"),
            pb.array("phi_minus"))

    def mesh_desc(self):
        return self.desc

    def array(self, name):
        assert name == "U0"
        return self.U


def problem(vt, nx, ny, p, io):
    return vt.Problem(vt.make_params(nx, ny, p=p, integration_order=io, perturb_grid=0.2), vt.vortex(epsilon=0.3))


def orders(K):
    return {"random": np.random.default_rng(5).permutation(K), "rolled": np.roll(np.arange(K), 1)}


# resident (at most 148 tiles) and launched
@pytest.mark.parametrize("nx,ny,p,io", [(3, 32, 3, 10), (3, 31, 2, 6), (3, 32, 1, 4), (3, 700, 0, 2), (3, 3200, 2, 4)])
@pytest.mark.parametrize("mapping", [0, 1])
def test_three_columns_alone_and_in_a_batch(vt, nx, ny, p, io, mapping):
    import ctypes
    pb = problem(vt, nx, ny, p, io)
    s, b = vt.Solver(pb), vt.Batch([pb])
    s.stage_mapping = mapping
    assert vt.lib().vt_batch_set_mapping(b._h, (ctypes.c_int * 1)(mapping)) == 0
    dt = small_dt(nx, ny, p)
    b.set_dt([dt])
    s.rk4(dt, 7)
    b.rk4(7)
    np.testing.assert_array_equal(s.download(), b.download(0))
    s.close()
    b.close()


@pytest.mark.parametrize("nx,ny,p,io", [(16, 12, 3, 10), (30, 20, 2, 5), (24, 24, 1, 8), (20, 16, 0, 2), (80, 70, 1, 4)])
@pytest.mark.parametrize("order", ["random", "rolled"])
def test_another_order_of_the_elements(vt, nx, ny, p, io, order):
    """The elements in another order are the same mesh. Which side evaluates a
    face depends on the order, so states agree to rounding: a few times 1e-16 of
    the state per step and term, against 1e-12 of it."""
    pb = problem(vt, nx, ny, p, io)
    m = Reordered(vt, pb, orders(pb.K)[order])
    s, r, b = vt.Solver(pb), vt.Solver((m.desc, m.keep)), vt.Batch([m])
    r.upload(m.U)
    dt, size = small_dt(nx, ny, p), np.abs(m.U).max()
    b.set_dt([dt])
    for x in (s, r):
        x.rk4(dt, 10)
    b.rk4(10)
    np.testing.assert_array_equal(r.download(), b.download(0))
    np.testing.assert_allclose(r.download(), s.download()[m.perm], rtol=0, atol=1e-12 * size)
    s.forward_euler(0.01 * dt, 3)
    r.forward_euler(0.01 * dt, 3)
    np.testing.assert_allclose(r.download(), s.download()[m.perm], rtol=0, atol=1e-12 * size)
    for x in (s, r, b):
        x.close()


@pytest.mark.parametrize("nx,ny,p,io,order", [(3, 32, 3, 10, None), (3, 31, 2, 6, None), (3, 32, 0, 2, None),
                                              (30, 20, 3, 8, "random"), (30, 20, 2, 5, "rolled"),
                                              (80, 70, 1, 4, "random"), (20, 16, 0, 2, "random")])
@pytest.mark.parametrize("reflect", [True, False])
def test_derivatives(vt, nx, ny, p, io, order, reflect):
    """<W, R' V> = <R'^T W, V> to 1e-12 of the root of the sum of squares of the
    terms (at most 500 roundings of 1.1e-16 each, independent of each other),
    and R' V agrees with the structured order's to the rounding of its terms."""
    pb = problem(vt, nx, ny, p, io)
    stiff = pb.array("stiff_ref").copy()
    if not reflect:
        stiff[0] *= 1.25
    perm = np.arange(pb.K) if order is None else orders(pb.K)[order]
    m = Reordered(vt, pb, perm, stiff)
    r = vt.Solver((m.desc, m.keep))
    rng = np.random.default_rng(nx)
    V = rng.standard_normal(m.U.shape) * np.abs(m.U).max(axis=(0, 1))
    W = rng.standard_normal(m.U.shape)
    JV = r.rhs_jvp(m.U, V)
    a, b = W * JV, V * r.rhs_vjp(m.U, W)
    assert abs(a.sum() - b.sum()) <= 1e-12 * np.sqrt((a ** 2).sum() + (b ** 2).sum())
    same = Reordered(vt, pb, np.arange(pb.K), stiff)
    s = vt.Solver((same.desc, same.keep))
    back = np.empty_like(V)
    back[perm] = V
    want = s.rhs_jvp(same.U, back)
    np.testing.assert_allclose(JV, want[perm], rtol=0, atol=1e-12 * np.abs(want).max())
    r.close()
    s.close()


def test_gradient(vt):
    """A checkpointed gradient in random order, against the structured order's."""
    pb = problem(vt, 24, 20, 2, 6)
    m = Reordered(vt, pb, orders(pb.K)["random"])
    s, r = vt.Solver(pb), vt.Solver((m.desc, m.keep))
    r.upload(m.U)
    lam = np.random.default_rng(1).standard_normal((pb.K, pb.Np, 4))
    dt = small_dt(24, 20, 2)
    want = s.adjoint_rk4(dt, 12, 3, lam)[m.perm]
    got = r.adjoint_rk4(dt, 12, 3, np.ascontiguousarray(lam[m.perm]))
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-11 * np.abs(want).max())
    r.close()
    s.close()


def test_batches_made_in_a_row(vt):
    """A batch's set-up is ordered on its own stream: what it learns about its
    lists does not depend on when the default stream's work is done."""
    import torch
    pb = problem(vt, 80, 70, 1, 4)
    m = Reordered(vt, pb, orders(pb.K)["random"])
    dt = small_dt(80, 70, 1)
    r = vt.Solver((m.desc, m.keep))
    r.upload(m.U)
    r.rk4(dt, 3)
    want = r.download()
    busy = torch.zeros(1 << 26, dtype=torch.float64, device="cuda")
    for _ in range(12):
        busy.add_(1.0)  # work under way on the default stream
        b = vt.Batch([m])
        b.set_dt([dt])
        b.rk4(3)
        np.testing.assert_array_equal(b.download(0), want)
        b.close()
    r.close()
