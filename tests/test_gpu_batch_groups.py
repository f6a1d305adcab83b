"""A batch of several small groups replays a captured step: the same steps as
single solvers make, bit for bit, whatever changed since the capture."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def small_dt(n, p):
    return 0.3 * 10.0 / n / ((2 * p + 1) * 17.0)


@pytest.mark.parametrize("n", [1, 5, 20])
def test_batch_of_many_small_groups(vt, n):
    shapes = [(8, 8, 1, 4), (5, 7, 2, 4), (24, 20, 2, 6), (4, 4, 3, 6), (9, 6, 3, 8), (8, 8, 1, 4)]
    pbs = [vt.Problem(vt.make_params(nx, ny, p=p, integration_order=io, perturb_grid=0.1),
                      vt.vortex(epsilon=0.2 + 0.02 * i)) for i, (nx, ny, p, io) in enumerate(shapes)]
    dts = [small_dt(max(nx, ny), p) for nx, ny, p, _ in shapes]
    b = vt.Batch(pbs)
    assert len(b.groups) == 5
    singles = [vt.Solver(pb) for pb in pbs]

    def steps():
        b.rk4(n)
        for i, s in enumerate(singles):
            s.rk4(dts[i], n)
            np.testing.assert_array_equal(b.download(i), s.download())

    b.set_dt(dts)
    for _ in range(11 if n == 1 else 3):
        steps()
    dts = [0.5 * dt for dt in dts]  # the time steps are not the graph's
    b.set_dt(dts)
    steps()
    groups = list(dict.fromkeys((p, io) for _, _, p, io in shapes))
    choice = b.autotune(trials=1)  # the groups' kernels and grids change
    for (_, _, p, io), s in zip(shapes, singles):
        s.stage_mapping = choice[groups.index((p, io))][1]
    steps()
    steps()
    b.close()
    for s in singles:
        s.close()
