"""A view factor of zero is +0 on every path, as raw / A of a sum of nothing is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nquad", [2, 4])
@pytest.mark.parametrize("kind", ["plates", "cube", "box", "cylinder", "cavity"])
def test_zeros_are_positive(rvf, session, kind, nquad, precision):
    from rvf_b200 import _abi
    M, obs = rvf.meshes, []
    if kind == "plates":
        md = M.parallel_plates(6, "quad4")
    elif kind == "cube":
        md = M.cube_enclosure(4, box=False)
    elif kind == "box":
        md, obs = M.cube_enclosure(4, box_m=3, box_edge=0.5), [7]
    elif kind == "cylinder":
        md = M.cylinder(nc=8, na=3, cap_rings=2)
    else:
        md, obs = M.cavity_2d(n_wall=20, n_circle=16, n_circles=2), [5, 6]
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, obs))
    try:
        F = np.empty((md.n_elems,) * 2, order="F")
        dm.solve(rvf.make_options(nquad, precision=precision, geometric_soup=True, seed=0), F)
    finally:
        dm.release()
    assert (F == 0.0).any()
    assert not np.signbit(F).any()
