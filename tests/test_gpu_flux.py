"""The device formulas of the face phase against IEEE arithmetic on the host,
and the stage kernel's folded operators against its unfolded ones."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_flux_formulas_match_ieee(tmp_path):
    """rsqrt_nr: series truncation below 0.02 ulp, five roundings in the
    correction of which only the last two weigh fully: two ulps. roe_flux2: each
    of about 60 dependent roundings of 1.1e-16 acts on a term no larger than the
    sizes it is compared with, some of them through the squares c2^2 and y^2:
    bounded by 2e-14 of them. The codes of the planted bad states are equal."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "gpu_flux_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "vortex-transport_b200", "csrc"),
                    os.path.join(ROOT, "tests", "gpu_flux_check.cu"), "-o", exe],
                   check=True, capture_output=True, text=True, timeout=600)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    m = dict(re.findall(r"(\w+) ([\d.e+-]+)", out))
    assert int(m["states"]) == 1 << 18 and int(m["bad"]) > 10000, out
    assert int(m["general"]) > 1000 and int(m["entropy_fixed"]) > 1000, out
    assert int(m["wrong_codes"]) == 0, out
    assert float(m["rsqrt_ulp"]) <= 2.0, out
    assert float(m["flux_rel"]) <= 2e-14, out
    print(out.strip())


@pytest.mark.parametrize("p,io,nx,ny", [(1, 2, 5, 4), (1, 5, 16, 4), (2, 4, 7, 3), (2, 10, 32, 6), (3, 6, 16, 2),
                                        (3, 8, 9, 5), (3, 19, 48, 4)])
def test_folded_operators_match_unfolded(vt, p, io, nx, ny):
    """Both forms of the stage kernel sum the same products, in another order:
    the right-hand sides agree to the rounding of their terms. A term is at
    most about max |D| max |G| (the volume) or max |lift| max |F| len/detJ (the
    surface), each sum has 2 Np or 3 nfq of them, and each addition rounds at
    1.1e-16."""
    pb = vt.Problem(vt.make_params(nx, ny, p=p, integration_order=io, perturb_grid=0.2))
    s = vt.Solver(pb)
    assert s.stage_mapping == 1
    folded = s.rhs()
    s.stage_mapping = 0
    plain = s.rhs()
    F = np.abs(pb.array("F0")).max()
    D = np.abs(np.einsum("ij,djk->dik", pb.array("minv_ref"), pb.array("stiff_ref"))).max()
    lift = np.abs(np.einsum("ij,sjq->siq", pb.array("minv_ref"), pb.array("phi_plus")) * pb.array("line_quad")[:, 1]).max()
    size = (2 * pb.Np * D * np.abs(pb.array("jinv")).max() * 2 * F
            + 3 * pb.nfq * lift * 20 * F * (pb.array("sides").max() / pb.array("detj").min()))
    assert np.abs(folded - plain).max() <= 8 * 1.1e-16 * size
    s.close()


def test_operators_without_the_symmetry(vt):
    """A caller's own tables need not be symmetric under xi <-> eta: both
    mappings then run the unfolded operators and agree bit for bit."""
    pb = vt.Problem(vt.make_params(16, 4, p=2, integration_order=6, perturb_grid=0.1))
    stiff = pb.array("stiff_ref").copy()
    stiff[1] *= 1.0 + 1e-6
    d, keep = vt.mesh_desc_from_arrays(2, pb.array("type"), pb.array("conn"), pb.array("detj"), pb.array("jinv"),
                                       pb.array("normals"), pb.array("sides"), pb.array("minv_ref"), stiff,
                                       pb.array("line_quad"), pb.array("phi_plus"), pb.array("phi_minus"))
    s = vt.Solver((d, keep))
    s.upload(pb.array("U0"))
    one = s.rhs()
    s.stage_mapping = 0
    two = s.rhs()
    s.close()
    s = vt.Solver(pb)
    base = s.rhs()
    s.close()
    scale = np.abs(base).max()
    assert np.abs(one - two).max() <= 1e-12 * max(scale, np.abs(one).max())
    assert np.abs(one - base).max() > 1e-9 * scale  # the caller's table was used
