"""Curves whose tiles or rows reach more segments than the curve kernel's lists hold
(kernels_occ2d.cu): their pairs are deferred to the queue pipeline.  Against the queue
pipeline alone (1e-12: the order of the sums; the same counts), the oracle, a
server's request and a session of little memory (the same bits)."""
import numpy as np
import pytest

from test_gpu_occ2d import solve
from test_gpu_parity import assert_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_wall,n_circle,n_circles,nquad", [
    (2, 60, 4, 3), (4, 60, 4, 8), (1, 200, 4, 2), (9, 333, 4, 4), (3, 900, 4, 1)])
def test_deferred(rvf, orc, session, n_wall, n_circle, n_circles, nquad):
    md = rvf.meshes.cavity_2d(n_wall=n_wall, n_circle=n_circle, n_circles=n_circles, seed=2)
    obs = list(range(5, 5 + n_circles))
    F, st = solve(rvf, session, md, nquad, obs)
    assert st["ms_resolve"] > 0.0, "no pair was deferred"
    Fq, stq = solve(rvf, session, md, nquad, obs, cull=False)
    for k in ("n_rays", "n_point_pairs"):
        assert st[k] == stq[k]
    assert_rel(F, Fq, rtol=1e-12)
    if md.n_elems <= 1500:
        raw, area, _, _ = orc.solve_plain(orc.Mesh(md, obs), nquad)
        assert_rel(F, orc.f_from_raw(raw, area))


def test_served_and_small_budget(rvf, session):
    from rvf_b200 import _abi
    md = rvf.meshes.cavity_2d(n_wall=4, n_circle=120, n_circles=4, seed=2)
    obs = [5, 6, 7, 8]
    F, st = solve(rvf, session, md, 4, obs)
    sv = _abi.Server(session)
    try:
        ids = [sv.submit(rvf.mesh_desc_arrays(md, obs), rvf.make_options(4, seed=0)) for _ in range(3)]
        for rid in ids:
            sv.wait(rid, 60000)
            assert np.array_equal(sv.result(rid)[0], F, equal_nan=True)
            sv.release(rid)
    finally:
        sv.close()
    own = rvf.Session(0, hbm_budget_bytes=24 << 20)
    try:
        Fs, sts = solve(rvf, own, md, 4, obs)
        assert np.array_equal(Fs, F, equal_nan=True) and sts["n_rays"] == st["n_rays"]
    finally:
        own.close()
