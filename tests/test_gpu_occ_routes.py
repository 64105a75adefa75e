"""Which kernels take the tiles with ray work (occ_by_queue, wave_host.cpp), on both
sides of its lines, and that either gives the oracle's view factors: obstructions
fine beside the elements, rules of few and of many points, few and many tiles."""
import numpy as np
import pytest

from test_gpu_parity import assert_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,m,box_m,nquad,precision,geometric,queue", [
    ("quad4", 8, 24, 1, "fp64", False, True), ("quad4", 8, 3, 1, "fp64", False, False),
    ("quad4", 8, 24, 2, "fp64", True, True), ("tri3", 2, 10, 3, "fp64", False, True),
    ("tri3", 2, 4, 3, "fp64", False, False), ("quad4", 8, 24, 3, "fp64", False, False),
    ("quad4", 12, 24, 2, "mixed", False, True), ("quad4", 12, 6, 2, "mixed", False, False),
    ("quad4", 12, 24, 3, "mixed", True, True), ("quad4", 4, 24, 3, "mixed", False, False)])
def test_route(rvf, orc, session, family, m, box_m, nquad, precision, geometric, queue):
    from rvf_b200 import _abi
    md = rvf.meshes.cube_enclosure(m, family=family, box_m=box_m, box_edge=0.4)
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, [7]))
    try:
        F = np.empty((md.n_elems,) * 2, order="F")
        st = dm.solve(rvf.make_options(nquad, precision=precision, geometric_soup=geometric, seed=0), F).as_dict()
    finally:
        dm.release()
    assert (st["ms_resolve"] > 0.0) == queue  # a phase of the queue pipeline alone
    raw, area, _, cnt = orc.solve_plain(orc.Mesh(md, [7]), nquad, geometric=geometric)
    Fo = orc.f_from_raw(raw, area)
    if precision == "fp64":
        assert_rel(F, Fo)
    else:
        assert np.max(np.abs(F - Fo)) <= 1e-6


@pytest.mark.parametrize("family,m,jitter,nquad,precision,geometric,queue", [
    ("quad4", 12, 0.0, 3, "mixed", True, True), ("tri3", 9, 0.0, 2, "mixed", True, True),
    ("quad", 8, 0.0, 3, "mixed", True, True), ("quad4", 12, 0.3, 3, "mixed", True, False),
    ("quad4", 12, 0.0, 3, "mixed", False, False), ("quad4", 12, 0.0, 3, "fp64", True, False),
    ("quad4", 12, 0.0, 4, "mixed", True, False)])
def test_route_along_the_axes(rvf, orc, session, family, m, jitter, nquad, precision, geometric, queue):
    """Structured meshes along the axes (fp64_rays_many), whose rays FP32 often cannot certify."""
    from rvf_b200 import _abi
    md = rvf.meshes.cube_enclosure(m, family=family, box_m=3, jitter=jitter)
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, [7]))
    try:
        F = np.empty((md.n_elems,) * 2, order="F")
        st = dm.solve(rvf.make_options(nquad, precision=precision, geometric_soup=geometric, seed=0), F).as_dict()
    finally:
        dm.release()
    assert (st["ms_resolve"] > 0.0) == queue
    raw, area, _, cnt = orc.solve_plain(orc.Mesh(md, [7]), nquad, geometric=geometric)
    Fo = orc.f_from_raw(raw, area)
    if precision == "fp64":
        assert_rel(F, Fo)
    else:
        assert np.max(np.abs(F - Fo)) <= 1e-6
