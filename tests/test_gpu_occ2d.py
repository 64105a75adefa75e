"""The curve occlusion kernel (kernels_occ2d.cu) against the oracle (1e-10
relative, the FP64 path's tolerance) and the queue pipeline (1e-12: the order
of the sums): one tile and partial ones, rules of 1 to 32 points, Line2, tiles
with few segments in reach and with more than a tile's list holds (every ray
walks the tree), walls that are obstructions themselves (own groups skipped)."""
import numpy as np
import pytest

from test_gpu_parity import assert_rel

pytestmark = pytest.mark.gpu


def solve(rvf, session, md, nquad, obs, cull=True):
    from rvf_b200 import _abi
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, obs))
    try:
        N = md.n_elems
        o = rvf.make_options(nquad, seed=0)
        o.disable_tile_cull = 0 if cull else 1
        F = np.empty((N, N), order="F")
        return F, dm.solve(o, F).as_dict()
    finally:
        dm.release()


@pytest.mark.parametrize("n_wall,n_circle,n_circles,nquad,obs", [
    (4, 8, 1, 1, [5]), (6, 8, 2, 2, [5, 6]), (24, 16, 2, 4, [5, 6]), (20, 60, 3, 3, [5, 6, 7]),
    (16, 200, 2, 2, [5, 6]), (10, 300, 4, 2, [5, 6, 7, 8]), (24, 16, 2, 3, [1, 3, 5]), (5, 12, 1, 32, [5])])
def test_cavity(rvf, orc, session, n_wall, n_circle, n_circles, nquad, obs):
    md = rvf.meshes.cavity_2d(n_wall=n_wall, n_circle=n_circle, n_circles=n_circles, seed=4)
    F, st = solve(rvf, session, md, nquad, obs)
    Fq, stq = solve(rvf, session, md, nquad, obs, cull=False)
    assert st["n_rays"] == stq["n_rays"] and st["n_point_pairs"] == stq["n_point_pairs"]
    assert_rel(F, Fq, rtol=1e-12)
    if nquad <= 16:  # the oracle's line rules end between 16 and 24 points
        raw, area, _, _ = orc.solve_plain(orc.Mesh(md, obs), nquad)
        assert_rel(F, orc.f_from_raw(raw, area))


def test_line2(rvf, orc, session):
    md = rvf.meshes.cavity_2d(n_wall=12, n_circle=20, n_circles=2, seed=5)
    en = md.elem_nodes.copy()
    en[:, 2:] = 0
    md = rvf.MeshData(md.coords, en, np.full(md.n_elems, 5, dtype=np.int8), md.elem_group, dict(md.group_tags),
                      dict(md.group_tri_soup), 1)
    F, _ = solve(rvf, session, md, 3, [5, 6])
    raw, area, _, _ = orc.solve_plain(orc.Mesh(md, [5, 6]), 3)
    assert_rel(F, orc.f_from_raw(raw, area))
