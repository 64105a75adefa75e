"""Monte Carlo on curves among more segments than a tile's list holds (claims of
eight rows, rows that walk the tree): the oracle's samples, decisions and view
factors bit for bit, below and above the list's 2,048."""
import pytest

from test_gpu_mc import assert_same, device_mc, oracle_mc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_wall,n_circle,n_circles,n", [(2, 512, 4, 2), (2, 513, 4, 2), (40, 700, 3, 1)])
def test_many_segments(rvf, orc, session, n_wall, n_circle, n_circles, n):
    md = rvf.meshes.cavity_2d(n_wall=n_wall, n_circle=n_circle, n_circles=n_circles, seed=3)
    obs = list(range(5, 5 + n_circles))
    F, A, _, st = device_mc(rvf, session, md, n, 9, obs)
    Fo, Ao, _, cnt = oracle_mc(orc, md, n, 9, obs)
    assert_same(A, Ao)
    assert_same(F, Fo)
    assert st.n_rays == cnt[1]
