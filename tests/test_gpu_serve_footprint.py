"""What the server charges a request for at admission covers the reductions'
buffer as it is allocated (at most 64 partial sums a row and group), not more: a
mesh of many groups is admitted within a budget that holds it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_many_groups(rvf, session):
    from rvf_b200 import _abi
    md = rvf.meshes.cube_enclosure(15, family="quad4", box=False)
    N, G = md.n_elems, 100
    md.elem_group[:] = 1 + np.arange(N) % G
    md.group_tags = {g: f"g{g}" for g in range(1, G + 1)}
    md.group_tri_soup = {}
    need = 8 * 64 * G * N + 8 * N * N
    sv = _abi.Server(session, admit_bytes=2 * need)
    try:
        rid = sv.submit(rvf.mesh_desc_arrays(md, []), rvf.make_options(2, seed=0))
        sv.wait(rid, 60000)
        F, A, Fg, Ag = sv.result(rid)
        assert Fg.shape == (G, G)
        assert need <= sv.stats()["admitted_bytes_peak"] <= 1.5 * need
        sv.release(rid)
    finally:
        sv.close()
