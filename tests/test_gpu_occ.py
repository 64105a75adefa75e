"""The occlusion kernels (kernels_occ.cu) against the oracle and the queue
pipeline (the same solve without tile classes).

Ray decisions are the oracle's, so FP64 agrees with it to 1e-10 relative and
with the queue pipeline to 1e-12 (only the order of the sums differs); mixed
precision to its 1e-6.  Sizes: one tile and a partial one, rules from 1 to 64
points (the lanes of a warp hold 64 rays at a time), lists beyond a row's 32
leaves and tiles beyond the kernels' 2,048 triangles (the pairs' own walks),
and a tree walked by every ray."""
import numpy as np
import pytest

from test_gpu_parity import assert_rel

pytestmark = pytest.mark.gpu


def solve(rvf, session, md, nquad, precision="fp64", cull=True, lists=True, geometric=False):
    from rvf_b200 import _abi
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, [7]))
    try:
        N = md.n_elems
        o = rvf.make_options(nquad, precision=precision, geometric_soup=geometric, seed=0)
        o.disable_tile_cull = 0 if cull else 1
        o.disable_pair_lists = 0 if lists else 1
        F = np.empty((N, N), order="F")
        st = dm.solve(o, F)
        return F, st.as_dict()
    finally:
        dm.release()


def check(rvf, orc, session, md, nquad, geometric, walk=False):
    F, st = solve(rvf, session, md, nquad, geometric=geometric)
    Fq, stq = solve(rvf, session, md, nquad, cull=False, geometric=geometric)
    assert st["n_rays"] == stq["n_rays"]
    assert_rel(F, Fq, rtol=1e-12)
    raw, area, _, _ = orc.solve_plain(orc.Mesh(md, [7]), nquad, geometric=geometric)
    Fo = orc.f_from_raw(raw, area)
    assert_rel(F, Fo)
    M, stm = solve(rvf, session, md, nquad, precision="mixed", geometric=geometric)
    assert stm["n_rays"] == st["n_rays"]
    assert np.max(np.abs(M - Fo)) <= 1e-6
    if walk:
        W, stw = solve(rvf, session, md, nquad, lists=False, geometric=geometric)
        assert stw["n_list_pairs"] == 0 and stw["n_walk_pairs"] == st["n_list_pairs"] + st["n_walk_pairs"]
        assert np.array_equal(W, F, equal_nan=True)
    return st


@pytest.mark.parametrize("geometric", [False, True])
@pytest.mark.parametrize("family,nquad", [("tri3", 1), ("tri3", 2), ("tri", 3), ("tri3", 4), ("quad4", 2), ("quad", 3),
                                          ("quad4", 4), ("quad", 5), ("quad4", 6), ("quad4", 8)])
def test_rules(rvf, orc, session, family, nquad, geometric):
    md = rvf.meshes.cube_enclosure(2 if family.startswith("tri") else 3, family=family, box_m=3, box_edge=0.5)
    check(rvf, orc, session, md, nquad, geometric, walk=nquad <= 3)


@pytest.mark.parametrize("m", [1, 4, 7])
def test_tile_edges(rvf, orc, session, m):
    """12, 192 and 588 elements: one partial tile, whole tiles, a remainder of 12."""
    check(rvf, orc, session, rvf.meshes.cube_enclosure(m, box_m=4, box_edge=0.4), 2, True)


@pytest.mark.parametrize("geometric", [False, True])
def test_long_lists(rvf, orc, session, geometric):
    """Elements larger than the box of 3,072 triangles: the tiles' and the pairs' lists overflow."""
    md = rvf.meshes.cube_enclosure(2, jitter=0.1, box_m=16, box_edge=0.5)
    st = check(rvf, orc, session, md, 2, geometric)
    assert st["n_list_pairs"] + st["n_walk_pairs"] > 0
