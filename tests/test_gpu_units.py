"""Meshes in small units or far from the origin, where FP32 coordinates are coarse
beside the obstruction's triangles (fp32_too_coarse, wave_host.cpp): the queue
pipeline takes them; on both sides of the line the oracle's view factors."""
import numpy as np
import pytest

from test_gpu_parity import assert_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geometric", [False, True])
@pytest.mark.parametrize("scale,offset,queue", [(1.0, 0.0, False), (1e3, 0.0, False), (1e-2, 0.0, False),
                                                (1e-4, 0.0, True), (1.0, 1e5, True)])
def test_scales_and_offsets(rvf, orc, session, scale, offset, queue, geometric):
    from rvf_b200 import _abi
    md = rvf.meshes.cube_enclosure(4, box_m=3, box_edge=0.4)
    shift = offset * np.array([0.6, -0.7, 0.4])
    md.coords[...] = md.coords * scale + shift[:, None]
    md.group_tri_soup[7] = md.group_tri_soup[7] * scale + shift
    raw, area, _, _ = orc.solve_plain(orc.Mesh(md, [7]), 3, geometric=geometric)
    Fo = orc.f_from_raw(raw, area)
    # elements in one plane: cosines of the coordinates' rounding
    same = np.asarray(md.elem_group)[:, None] == np.asarray(md.elem_group)[None, :]
    for precision in ("fp64", "mixed"):
        dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, [7]))
        try:
            F = np.empty((md.n_elems,) * 2, order="F")
            st = dm.solve(rvf.make_options(3, precision=precision, geometric_soup=geometric, seed=0), F).as_dict()
        finally:
            dm.release()
        assert (st["ms_resolve"] > 0.0) == queue
        if precision == "fp64":
            assert_rel(np.where(same, 0.0, F), np.where(same, 0.0, Fo))
        elif offset == 0.0:
            assert np.max(np.abs(F - Fo)) <= 1e-6


@pytest.mark.parametrize("scale,nquad,queue", [(1.0, 2, False), (1e3, 2, True), (1e3, 3, False)])
def test_large_units(rvf, orc, session, scale, nquad, queue):
    """Millimetres: the margin of the lists' triangle test exceeds the triangles, and rules of few points
    among many leaves are taken by the queue pipeline (occ_by_queue)."""
    from rvf_b200 import _abi
    md = rvf.meshes.cube_enclosure(12, box_m=12)
    md.coords[...] *= scale
    md.group_tri_soup[7] = md.group_tri_soup[7] * scale
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, [7]))
    try:
        F = np.empty((md.n_elems,) * 2, order="F")
        st = dm.solve(rvf.make_options(nquad, seed=0), F).as_dict()
    finally:
        dm.release()
    assert (st["ms_resolve"] > 0.0) == queue
    raw, area, _, _ = orc.solve_plain(orc.Mesh(md, [7]), nquad)
    assert_rel(F, orc.f_from_raw(raw, area))
