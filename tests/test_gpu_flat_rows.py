"""Plane pairs in the quadrature-only kernel (flat_rows): rules of 1 to 7 points,
partial tiles, plane and curved elements, pairs too near or too grazing for the plane
loop.  F equals that of single-row tasks, which run the general kernel, bit for bit,
and the oracle's to 1e-10."""
import numpy as np
import pytest

from test_gpu_parity import assert_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,nquad", [("tri3", 1), ("tri3", 2), ("tri3", 3), ("tri", 2), ("tri", 3), ("quad4", 1),
                                          ("quad4", 2), ("quad", 2)])
@pytest.mark.parametrize("mesh", ["plates", "cube", "cylinder", "cube+box"])
def test_rows(rvf, orc, session, family, nquad, mesh):
    from rvf_b200 import _abi
    M = rvf.meshes
    obs = []
    if mesh == "plates":
        md = M.parallel_plates(9, family)
    elif mesh == "cylinder":
        md = M.cylinder(nc=16, na=6, cap_rings=2, seed=3)
    else:
        obs = [7] if mesh == "cube+box" else []
        md = M.cube_enclosure(9 if family in ("quad4", "quad") else 7, family=family, box=bool(obs), box_m=2)
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, obs))
    try:
        N = md.n_elems
        got = {}
        for groups in (1, 2, 8, 32):
            o = rvf.make_options(nquad, seed=0)
            o.fast_row_groups = groups
            F = np.empty((N, N), order="F")
            st = dm.solve(o, F).as_dict()
            got[groups] = F, st["n_point_pairs"], st["n_rays"]
    finally:
        dm.release()
    for groups in (1, 2, 8):
        assert np.array_equal(got[groups][0], got[32][0], equal_nan=True), groups
        assert got[groups][1:] == got[32][1:], groups
    raw, area, _, _ = orc.solve_plain(orc.Mesh(md, obs), nquad)
    assert_rel(got[1][0], orc.f_from_raw(raw, area))
