"""The reverse stage with operators that have no reflection symmetry (a caller's
own tables): one launch over the tiles, as with the reference's, so no face
adjoints are kept in memory, and the same transpose."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solver(vt, nx, ny, p, io, factor):
    pb = vt.Problem(vt.make_params(nx, ny, p=p, integration_order=io, perturb_grid=0.2), vt.vortex(epsilon=0.3))
    stiff = pb.array("stiff_ref").copy()
    stiff[0] *= factor
    s = vt.Solver(vt.mesh_desc_from_arrays(pb.p, pb.array("type"), pb.array("conn"), pb.array("detj"), pb.array("jinv"),
                                           pb.array("normals"), pb.array("sides"), pb.array("minv_ref"), stiff,
                                           pb.array("line_quad"), pb.array("phi_plus"), pb.array("phi_minus")))
    U = pb.array("U0")
    s.upload(U)
    return s, U


def test_no_more_memory_than_with_the_reference_operators(vt):
    """11 state vectors: 34.6 MB here; the face adjoints of the two-launch form
    would add 25 MB. A driver allocates in pieces of at most 2 MB more."""
    import torch
    used = {}
    for factor in (1.0, 1.25):
        tiny, U = solver(vt, 4, 4, 1, 6, factor)
        tiny.rhs_vjp(U, np.ones_like(U))  # loads the kernels
        s, U = solver(vt, 128, 128, 1, 6, factor)
        W = torch.ones(U.shape, dtype=torch.float64, device="cuda")
        dU = torch.from_numpy(U).cuda()
        keep = torch.empty_like(W)  # the result's place in torch's pool
        del keep
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s.rhs_vjp(dU, W)
        used[factor] = before - torch.cuda.mem_get_info()[0]
        s.close()
        tiny.close()
    assert used[1.0] >= 11 * 6 * 2 * 128 * 128 * 16
    assert used[1.25] <= used[1.0] + (4 << 20), used


@pytest.mark.parametrize("nx,ny,p,io", [(4, 2, 3, 10), (9, 7, 3, 19), (16, 16, 2, 5), (40, 38, 1, 3), (12, 9, 0, 2),
                                        (150, 131, 2, 6)])
def test_gradient_transposes_the_tangent(vt, nx, ny, p, io):
    """<W, dU(T)> = <dJ/dU(0), dU(0)> over six steps. A step's tangent is four
    stages of sums of fewer than 500 products each; errors of different entries
    are independent, so 2e-12 of the root of the sum of squares holds six steps'
    worth of 500 eps = 1.1e-13 with room for the terms' excess over the entries."""
    s, U = solver(vt, nx, ny, p, io, 1.0 + 1e-3)
    rng = np.random.default_rng(nx)
    V = rng.standard_normal(U.shape) * np.abs(U).max(axis=(0, 1))
    W = rng.standard_normal(U.shape)
    dt = 0.1 * 10.0 / max(nx, ny) / ((2 * p + 1) * 17.0)
    dUT = s.tangent_rk4(dt, 6, V)
    s.upload(U)
    for snapshots in (2, 24):
        g = s.adjoint_rk4(dt, 6, snapshots, W)
        s.upload(U)
        a, b = W * dUT, V * g
        assert abs(a.sum() - b.sum()) <= 2e-12 * np.sqrt((a ** 2).sum() + (b ** 2).sum())
    s.close()
