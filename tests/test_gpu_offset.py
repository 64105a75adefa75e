"""FP64 quadrature of plane elements far from the origin, where the coordinates'
rounding is large beside the distances between planes: within the FP64 path's
1e-10 of the oracle, which integrates the same rounded coordinates."""
import numpy as np
import pytest

from test_gpu_parity import assert_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [False, True])
@pytest.mark.parametrize("family,nquad", [("tri3", 2), ("tri3", 3), ("quad4", 2), ("tri3", 4), ("quad4", 4)])
@pytest.mark.parametrize("offset", [0.0, 1e2, 1e3, 1e4, 1e5])
def test_translated(rvf, orc, session, offset, family, nquad, box):
    from rvf_b200 import _abi
    md = rvf.meshes.cube_enclosure(7, family=family, box=box, box_m=3)
    shift = offset * np.array([0.6, -0.7, 0.4])
    q, _ = np.linalg.qr(np.random.default_rng(1).normal(size=(3, 3)))
    md.coords[...] = q @ md.coords + shift[:, None]
    if box:
        md.group_tri_soup[7] = md.group_tri_soup[7] @ q.T + shift
    obs = [7] if box else []
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, obs))
    try:
        F = np.empty((md.n_elems,) * 2, order="F")
        dm.solve(rvf.make_options(nquad, geometric_soup=True, seed=0), F)
    finally:
        dm.release()
    raw, area, _, _ = orc.solve_plain(orc.Mesh(md, obs), nquad, geometric=True)
    # elements in one plane, whose cosines are the coordinates' rounding, are left out
    same = np.asarray(md.elem_group)[:, None] == np.asarray(md.elem_group)[None, :]
    Fo = orc.f_from_raw(raw, area)
    assert_rel(np.where(same, 0.0, F), np.where(same, 0.0, Fo))
