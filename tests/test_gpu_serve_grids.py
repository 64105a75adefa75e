"""The server's chunk grids are tuned for the queue pipeline alone: a class whose
tiles run in the occlusion kernels, which do not take them, reports the default."""
import pytest

pytestmark = pytest.mark.gpu


def test_reported_grids(rvf):
    from rvf_b200 import _abi
    own = rvf.Session(0)  # no choices of other tests
    sv = _abi.Server(own, max_batch=1)
    try:
        for precision in ("fp64", "mixed"):
            for _ in range(6):
                md = rvf.meshes.cube_enclosure(10, family="tri3", box_m=3)
                o = rvf.make_options(3, seed=0, precision=precision)
                rid = sv.submit(rvf.mesh_desc_arrays(md, [7]), o)
                sv.wait(rid, 120000)
                sv.release(rid)
        tuned = sv.stats()["tuned"]
    finally:
        sv.close()
        own.close()
    assert len(tuned) == 2
    assert [(t["gen_blocks_per_sm"], t["trace_blocks_per_sm"]) for t in tuned] == [(0, 0)] * 2
