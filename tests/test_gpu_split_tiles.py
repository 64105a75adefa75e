"""A solve whose list pool runs full (a small memory budget, long lists, tiles
claimed in parts): more chunks, the same view factors and the same counts as a
solve that holds every tile at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = ("n_point_pairs", "n_rays", "n_pairs_masked")


@pytest.mark.parametrize("m,box_m", [(5, 16), (6, 16), (8, 24)])
def test_counts_do_not_depend_on_the_budget(rvf, session, m, box_m):
    from rvf_b200 import _abi
    md = rvf.meshes.cube_enclosure(m, family="quad4", box_m=box_m, box_edge=0.9)
    opts = rvf.make_options(2, geometric_soup=True, seed=0)

    def solve(s):
        dm = _abi.DeviceMesh(s, rvf.mesh_desc_arrays(md, [7]))
        try:
            F = np.empty((md.n_elems,) * 2, order="F")
            return F, dm.solve(opts, F).as_dict()
        finally:
            dm.release()

    F0, st0 = solve(session)
    split = 0
    for mib in np.arange(4.0, 15.0, 0.5):
        s = rvf.Session(0, hbm_budget_bytes=int(mib * 2 ** 20))
        try:
            F, st = solve(s)
        except rvf.RVFError as e:
            assert "ENOMEM" in str(e) or "EBUDGET" in str(e), e
            continue
        finally:
            s.close()
        split += st["n_chunks"] > 1
        assert {k: st[k] for k in COUNTS} == {k: st0[k] for k in COUNTS}, (mib, st["n_chunks"])
        assert np.array_equal(F, F0, equal_nan=True)
    assert split > 0, "no budget split the solve"
