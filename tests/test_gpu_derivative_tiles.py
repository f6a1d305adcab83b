"""The derivative kernels where their tiles can go wrong: ragged last tiles, a
tile with more leaving faces than slots (one column of cells), more tiles than
the persistent grid has blocks, and operators that do not reflect under the
swap of xi and eta (the kernels then read the operators as they are, and the
reverse stage is two launches); and the batch's reverse sweep, which reads and
writes each instance at its place in the caller's array, with instances of
several groups in between and with arrays that start on an odd double."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solver(vt, nx, ny, p, io, reflect):
    pb = vt.Problem(vt.make_params(nx, ny, p=p, integration_order=io, perturb_grid=0.2), vt.vortex(epsilon=0.3, M_infty=0.5))
    if reflect:
        return vt.Solver(pb), pb.array("U0")
    stiff = pb.array("stiff_ref").copy()
    stiff[0] *= 1.25  # the two directions now differ by more than a swap of nodes
    desc = vt.mesh_desc_from_arrays(pb.p, pb.array("type"), pb.array("conn"), pb.array("detj"), pb.array("jinv"),
                                    pb.array("normals"), pb.array("sides"), pb.array("minv_ref"), stiff,
                                    pb.array("line_quad"), pb.array("phi_plus"), pb.array("phi_minus"))
    s = vt.Solver(desc)
    s.upload(pb.array("U0"))
    return s, pb.array("U0")


@pytest.mark.parametrize("nx,ny,p,io,reflect", [(5, 7, 3, 10, True), (1, 70, 3, 8, True), (1, 70, 0, 2, True),
                                                (33, 19, 2, 5, True), (131, 113, 1, 4, True), (131, 113, 3, 10, True),
                                                (131, 113, 3, 10, False), (9, 6, 2, 7, False), (1, 70, 1, 3, False)])
def test_vjp_transposes_jvp(vt, nx, ny, p, io, reflect):
    """<W, R' V> = <R'^T W, V>. An entry of either side is a sum of fewer than
    500 rounded products, so it is off by at most 500 eps = 1.1e-13 of the sum of
    their magnitudes. Those exceed the entry itself by less than ten on average
    (V and W are random, so the sums do not cancel), and the errors of different
    entries are independent: 1e-12 of the root of the sum of squares."""
    s, U = solver(vt, nx, ny, p, io, reflect)
    rng = np.random.default_rng(nx + ny)
    V = rng.standard_normal(U.shape) * np.abs(U).max(axis=(0, 1))
    W = rng.standard_normal(U.shape)
    a, b = W * s.rhs_jvp(U, V), V * s.rhs_vjp(U, W)
    assert abs(a.sum() - b.sum()) <= 1e-12 * np.sqrt((a ** 2).sum() + (b ** 2).sum())
    s.close()


@pytest.mark.parametrize("nx,ny,p,io,reflect", [(5, 7, 3, 10, True), (1, 70, 3, 8, True), (131, 113, 1, 4, True),
                                                (9, 6, 2, 7, False)])
def test_jvp_is_the_derivative_of_the_stage(vt, nx, ny, p, io, reflect):
    """Central differences with h = 1e-6 leave h^2 from the third derivative and
    eps/h = 2.2e-10 of the residual's terms, a few hundred times over: 1e-7."""
    s, U = solver(vt, nx, ny, p, io, reflect)
    V = np.random.default_rng(nx).standard_normal(U.shape) * np.abs(U).max(axis=(0, 1))
    JV, h = s.rhs_jvp(U, V), 1e-6
    s.upload(U + h * V)
    R = s.rhs()
    s.upload(U - h * V)
    fd = (R - s.rhs()) / (2 * h)
    np.testing.assert_allclose(JV, fd, rtol=0, atol=1e-7 * np.abs(fd).max())
    s.close()


@pytest.mark.parametrize("odd", [False, True])
def test_batch_reverse_sweep_in_place(vt, odd):
    import torch
    pbs = [vt.Problem(vt.make_params(nx, ny, p=p, integration_order=io, perturb_grid=0.1), vt.vortex(epsilon=0.3))
           for nx, ny, p, io in [(9, 7, 2, 5), (5, 6, 1, 4), (8, 8, 2, 5), (1, 40, 1, 4), (6, 5, 3, 10)]]
    b = vt.Batch(pbs)
    assert len(b.groups) == 3
    b.set_dt([2e-4] * len(pbs))
    b.adjoint_forward(5, 3)
    rng = np.random.default_rng(3)
    lams = [rng.standard_normal((pb.K, pb.Np, 4)) for pb in pbs]
    want = b.adjoint_backward(lams)  # host arrays
    n = sum(x.size for x in lams)
    src = torch.zeros(n + 2, dtype=torch.float64, device="cuda")
    out = torch.full((n + 2,), 7.0, dtype=torch.float64, device="cuda")
    at = 1 if odd else 0
    src[at:at + n] = torch.from_numpy(np.concatenate([x.ravel() for x in lams])).cuda()
    torch.cuda.synchronize()
    st = vt.lib().vt_batch_adjoint_backward_device(b._h, ctypes.c_void_p(src[at:].data_ptr()),
                                                   ctypes.c_void_p(out[at:].data_ptr()))
    assert st == 0
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[at:at + n], np.concatenate([x.ravel() for x in want]))
    assert (np.delete(got, np.arange(at, at + n)) == 7.0).all()
    b.close()
