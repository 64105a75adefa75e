"""Radiating elements that are obstructions too: an enclosure around a body, the body's
groups or all of them as obstruction.  Every ray to the body ends on its boxes, where
FP32 box tests are uncertain; few rays may need FP64 for that, and decisions and
counts are the oracle's."""
import numpy as np
import pytest

from test_gpu_parity import assert_rel

pytestmark = pytest.mark.gpu

REVERSED = {"tri3": [0, 2, 1], "quad4": [0, 3, 2, 1]}


def enclosure_with_body(rvf, family, m, m_body):
    a = rvf.meshes.cube_enclosure(m, family=family, box=False)
    b = rvf.meshes.cube_enclosure(m_body, family=family, box=False, seed=5)
    en = np.zeros_like(b.elem_nodes)
    en[:, :len(REVERSED[family])] = b.elem_nodes[:, REVERSED[family]] + a.coords.shape[1]
    soups = dict(a.group_tri_soup)
    md = rvf.MeshData(np.asfortranarray(np.hstack([a.coords, 0.3 * (b.coords - 0.5) + 0.5])),
                      np.vstack([a.elem_nodes, en]).astype(np.int32), np.concatenate([a.elem_family, b.elem_family]),
                      np.concatenate([a.elem_group, b.elem_group + 6]).astype(np.int32),
                      {g: f"g{g}" for g in range(1, 13)}, soups, 2)
    from rvf_b200.mesh import build_group_obs_soups
    md.group_tri_soup = {int(k): np.ascontiguousarray(v) for k, v in build_group_obs_soups(md).items()}
    return md


@pytest.mark.parametrize("geometric", [False, True])
@pytest.mark.parametrize("family,m,m_body,nquad,first", [("tri3", 5, 3, 3, 7), ("tri3", 4, 3, 4, 1), ("quad4", 6, 4, 3, 7),
                                                         ("quad4", 8, 5, 2, 1)])
def test_body(rvf, orc, session, family, m, m_body, nquad, first, geometric):
    from rvf_b200 import _abi
    md = enclosure_with_body(rvf, family, m, m_body)
    obs = list(range(first, 13))
    raw, area, _, _ = orc.solve_plain(orc.Mesh(md, obs), nquad, geometric=geometric)
    Fo = orc.f_from_raw(raw, area)
    rays = {}
    for precision in ("fp64", "mixed"):
        for cull in (0, 1):
            dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, obs))
            try:
                F = np.empty((md.n_elems,) * 2, order="F")
                o = rvf.make_options(nquad, precision=precision, geometric_soup=geometric, seed=0)
                o.disable_tile_cull = cull
                st = dm.solve(o, F).as_dict()
            finally:
                dm.release()
            rays[precision, cull] = st["n_rays"]
            if precision == "fp64":
                assert_rel(F, Fo)
            else:
                assert np.max(np.abs(F - Fo)) <= 1e-6
            # boxes touched at a ray's end no longer send it to FP64: few rays are left
            assert st["n_unsure_rays"] <= 0.05 * st["n_rays"]
    assert len(set(rays.values())) == 1
