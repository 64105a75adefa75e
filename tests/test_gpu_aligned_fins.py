"""Obstructions whose edges run along the pairs' directions: plates facing each
other with fins between them, turned off the axes, so that the directions and
edges are parallel only up to rounding.  Every shadow ray is decided as the
oracle decides it."""
import numpy as np
import pytest

from test_gpu_parity import assert_rel

pytestmark = pytest.mark.gpu


def fin(x, y0, y1, z0, z1, ny, nz):
    """ny x nz cells of two triangles in the plane at x."""
    y, z = np.linspace(y0, y1, ny + 1), np.linspace(z0, z1, nz + 1)
    tris = []
    for a in range(ny):
        for b in range(nz):
            c = [(x, y[a], z[b]), (x, y[a + 1], z[b]), (x, y[a + 1], z[b + 1]), (x, y[a], z[b + 1])]
            tris += [(c[0], c[1], c[2]), (c[0], c[2], c[3])]
    return np.asarray(tris)


def plates_with_fins(rvf, seed):
    rng = np.random.default_rng(seed)
    n = 10
    md = rvf.meshes.parallel_plates(n, "quad4")
    soup = np.concatenate([fin((k + rng.uniform(0.3, 0.7)) / n, 0.03, 0.97, 0.3, 0.7, 14, 3) for k in range(1, n, 2)])
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    q *= np.sign(np.linalg.det(q))
    md.coords[...] = q @ md.coords
    md.group_tri_soup[7] = np.ascontiguousarray(soup @ q.T)
    return md


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("geometric", [False, True])
@pytest.mark.parametrize("cull", [True, False])
def test_quadrature(rvf, orc, session, seed, cull, geometric):
    """cull: the occlusion kernels; without: the queue pipeline's lists."""
    from rvf_b200 import _abi
    md = plates_with_fins(rvf, seed)
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, [7]))
    try:
        F = np.empty((md.n_elems,) * 2, order="F")
        o = rvf.make_options(3, geometric_soup=geometric, seed=0)
        o.disable_tile_cull = 0 if cull else 1
        dm.solve(o, F)
    finally:
        dm.release()
    raw, area, _, _ = orc.solve_plain(orc.Mesh(md, [7]), 3, geometric=geometric)
    assert_rel(F, orc.f_from_raw(raw, area))


@pytest.mark.parametrize("seed", range(2))
def test_monte_carlo(rvf, orc, session, seed):
    from rvf_b200 import _abi
    md = plates_with_fins(rvf, seed)
    dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, [7]))
    try:
        F = np.empty((md.n_elems,) * 2, order="F")
        dm.solve(rvf.make_options(3, monte_carlo=True, n_samples=25, geometric_soup=True, seed=5), F)
    finally:
        dm.release()
    raw, area = orc.solve_mc(orc.Mesh(md, [7]), 25, 5, geometric=True)[:2]
    assert np.array_equal(F, orc.f_from_raw(raw, area), equal_nan=True)
