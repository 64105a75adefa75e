"""Monte Carlo kernels at the edges of their divisions: sample counts around the
32 that share a pair's lanes (and strata that are and are not powers of two), one
element to several tiles, every element family, lists that overflow.  Areas, ray
decisions and F equal the oracle's bit for bit."""
import numpy as np
import pytest

from test_gpu_mc import assert_same, device_mc, oracle_mc

pytestmark = pytest.mark.gpu


def same_as_oracle(rvf, orc, session, md, n, obs, exclude=True, blocked=True):
    F, A, lg, st = device_mc(rvf, session, md, n, 77, obs, exclude, log=True)
    Fo, Ao, lgo, cnt = oracle_mc(orc, md, n, 77, obs, exclude, log=True)
    assert np.array_equal(A, Ao)
    assert np.array_equal(lg, lgo), f"{int((lg != lgo).sum())} ray decisions differ"
    assert_same(F, Fo)
    assert st.n_rays == cnt[1]
    if blocked:
        assert (lgo == 2).sum() > 0


@pytest.mark.parametrize("n", [1, 2, 3, 4, 9, 31, 32, 33, 36, 64, 65])
def test_surface_samples(rvf, orc, session, n):
    md = rvf.meshes.cube_enclosure(3, family="quad4", box_m=2)
    same_as_oracle(rvf, orc, session, md, n, [7], blocked=n > 3)


@pytest.mark.parametrize("family", ["tri3", "tri", "quad4", "quad"])
@pytest.mark.parametrize("m", [1, 2, 4, 5])
def test_surface_families(rvf, orc, session, family, m):
    md = rvf.meshes.cube_enclosure(m, family=family, box_m=3)
    same_as_oracle(rvf, orc, session, md, 9, [7])


@pytest.mark.parametrize("n", [1, 2, 5, 33])
@pytest.mark.parametrize("n_wall,n_circle,n_circles,obs", [
    (4, 8, 1, [5]), (12, 16, 2, [5, 6]), (9, 300, 4, [5, 6, 7, 8]), (10, 1400, 2, [5, 6])])
def test_curves(rvf, orc, session, n, n_wall, n_circle, n_circles, obs):
    md = rvf.meshes.cavity_2d(n_wall=n_wall, n_circle=n_circle, n_circles=n_circles, seed=6)
    if md.n_elems * md.n_elems * n > 2e6:
        n = 1
    same_as_oracle(rvf, orc, session, md, n, obs, blocked=False)


@pytest.mark.parametrize("lift", [0.0, 0.25])
def test_line2(rvf, orc, session, lift):
    md = rvf.meshes.cavity_2d(n_wall=12, n_circle=20, n_circles=2, seed=5)
    en = md.elem_nodes.copy()
    en[:, 2:] = 0
    xyz = md.coords.copy()
    xyz[::3, 2] += lift  # nodes off the plane: the z terms count
    md = rvf.MeshData(xyz, en, np.full(md.n_elems, 5, dtype=np.int8), md.elem_group, dict(md.group_tags),
                      dict(md.group_tri_soup), 1)
    same_as_oracle(rvf, orc, session, md, 6, [5, 6])
