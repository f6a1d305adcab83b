"""Meshes whose neighbour tables are not mutual. vt_create takes any table with
ids in range; one launch per stage is right for all of them, many steps in one
launch only where the tiles read each other mutually, so the solver must not
use that form here. A batch always steps by a launch per stage: the same mesh
alone and as a batch of one agrees bit for bit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_mutual_tiles_are_recognised(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is not available")
    exe = str(tmp_path / "tile_reads_check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror",
                    "-I", os.path.join(ROOT, "vortex-transport_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "tile_reads_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.count("OK") == 7, out.stdout


class OneWay:
    """Two copies of a periodic mesh: the second on its own, the first with its
    leftmost cells reading the second's in place of their own neighbours."""

    def __init__(self, vt, nx, ny, p, io):
        pb = vt.Problem(vt.make_params(nx, ny, p=p, integration_order=io, perturb_grid=0.0), vt.vortex(epsilon=0.3))
        self.pb, self.K, self.Np, self.p = pb, 2 * pb.K, pb.Np, pb.p

        def twice(name):
            return np.concatenate([pb.array(name)] * 2)
        conn = np.concatenate([pb.array("conn"), pb.array("conn") + pb.K])
        first = np.arange(0, pb.K, 2 * nx)  # the type-0 element of every row's first cell
        conn[first, 1] += pb.K              # its left neighbour
        self.desc, self.keep = vt.mesh_desc_from_arrays(
            p, twice("type"), conn, twice("detj"), twice("jinv"), twice("normals"), twice("sides"),
            pb.array("minv_ref"), pb.array("stiff_ref"), pb.array("line_quad"), pb.array("phi_plus"), pb.array("phi_minus"))
        U = pb.array("U0")
        other = vt.Problem(vt.make_params(nx, ny, p=p, integration_order=io, perturb_grid=0.0),
                           vt.vortex(epsilon=0.15, x0=1.0, y0=-0.5))
        self.U = np.concatenate([U, other.array("U0")])

    def mesh_desc(self):
        return self.desc

    def array(self, name):
        assert name == "U0"
        return self.U


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,p,io", [(16, 12, 2, 6), (24, 20, 1, 4), (8, 24, 3, 10)])
@pytest.mark.parametrize("mapping", [0, 1])
def test_one_way_mesh_alone_and_in_a_batch(vt, nx, ny, p, io, mapping):
    import ctypes
    m = OneWay(vt, nx, ny, p, io)
    s, b = vt.Solver((m.desc, m.keep)), vt.Batch([m])
    s.upload(m.U)
    s.stage_mapping = mapping
    assert vt.lib().vt_batch_set_mapping(b._h, (ctypes.c_int * 1)(mapping)) == 0
    dt = 0.1 * 10.0 / max(nx, ny) / ((2 * p + 1) * 17.0)
    b.set_dt([dt])
    for n in (1, 60):
        s.rk4(dt, n)
        b.rk4(n)
        np.testing.assert_array_equal(s.download(), b.download(0))
    # the second copy goes its own way: it never reads the first
    alone = vt.Solver(m.pb)
    alone.upload(m.U[m.pb.K:])
    alone.rk4(dt, 61)
    np.testing.assert_allclose(s.download()[m.pb.K:], alone.download(), rtol=0, atol=1e-12 * np.abs(m.U).max())
    s.close()
    b.close()
    alone.close()
