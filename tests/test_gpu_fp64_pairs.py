"""The FP64 quadrature-only loops (device_pairs.cuh) against the oracle, at the
lines between their branches: plane elements far apart and near, cosines
around the plane loop's 1e-3 and the grazing test's 1e-5, rules of 1 to 64
points (full and partial point blocks), curved elements.  Tolerance: the FP64
path's 1e-10 relative."""
import numpy as np
import pytest

from test_gpu_parity import assert_rel

pytestmark = pytest.mark.gpu


def compare(rvf, orc, session, md, nquad):
    from rvf_b200 import _abi
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, []))
    try:
        N = md.n_elems
        F = np.empty((N, N), order="F")
        dm.solve(rvf.make_options(nquad, seed=0), F)
    finally:
        dm.release()
    raw, area, _, _ = orc.solve_plain(orc.Mesh(md), nquad)
    assert_rel(F, orc.f_from_raw(raw, area))


def tilted(rvf, family, n, cosine, gap):
    """Two plates side by side, the second one facing down and rising from the first one's plane with
    slope `cosine`: their points see one another at cosines around that value."""
    md = rvf.meshes.parallel_plates(n, family)
    up = md.coords[2] > 0.5
    md.coords[2, up] = cosine * (1.0 + md.coords[0, up])
    md.coords[0, up] += 1.0 + gap
    return md


@pytest.mark.parametrize("cosine", [0.0, 3e-6, 9.9e-6, 1.1e-5, 5e-4, 1.5e-3])
@pytest.mark.parametrize("family,nquad", [("quad4", 2), ("tri3", 3)])
def test_small_cosines(rvf, orc, session, family, nquad, cosine):
    compare(rvf, orc, session, tilted(rvf, family, 4, cosine, 0.25), nquad)


@pytest.mark.parametrize("gap", [0.02, 0.3, 2.5, 2.6, 8.0])
def test_near_and_far_plates(rvf, orc, session, gap):
    compare(rvf, orc, session, rvf.meshes.parallel_plates(5, "quad4", gap=gap), 3)


@pytest.mark.parametrize("family,nquad", [("tri3", 1), ("tri", 2), ("quad4", 2), ("tri3", 3), ("quad", 3), ("tri", 4),
                                          ("quad4", 4), ("quad4", 5), ("quad", 6), ("quad4", 7), ("quad", 8)])
def test_rules(rvf, orc, session, family, nquad):
    compare(rvf, orc, session, rvf.meshes.cube_enclosure(2, family=family, box=False), nquad)


def test_curved(rvf, orc, session):
    compare(rvf, orc, session, rvf.meshes.cylinder(nc=8, na=3, cap_rings=2, jitter=0.01, seed=3), 4)
