"""Mixed precision, elements that bulge far beyond their corners: two Quad8 domes
tip to tip, their centroids 480 times as far apart as the tips.  The direction of
the tips' ray, formed in FP32 from the centroids, is off by up to 3e-5, which the
triangle test's allowances must cover: the triangle between the tips is tilted
against the ray so little that its determinant (1.002e-10) barely passes the
reference's cut of 1e-10 (src/GPUBVH.jl:250), and blocks it.

The tips' term is all but 2e-5 of the unblocked view factor: a wrong decision is
off by four orders of magnitude."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, GAP, SIZE, EDGE, DET = 0.3, 0.001, 0.01, 1e-3, 1.002e-10


def domes(rvf, seed):
    rng = np.random.default_rng(seed)
    c = 0.5 * SIZE * np.array([(-1, -1), (1, -1), (1, 1), (-1, 1), (0, -1), (1, 0), (0, 1), (-1, 0)], float)
    z = np.array([0.0] * 4 + [H] * 4)
    top = [0, 3, 2, 1, 7, 6, 5, 4]
    p = np.vstack([np.column_stack([c, z]), np.column_stack([c[top], 4 * H + GAP - z[top]])])
    # the tips' ray runs along z from 2 H to 2 H + GAP, through the triangle's centroid
    tilt = (1 if seed % 2 else -1) * DET / EDGE ** 2
    e1, e2 = EDGE * np.array([0.0, np.sin(tilt), np.cos(tilt)]), EDGE * np.array([1.0, 0.0, 0.0])
    v0 = np.array([0.0, 0.0, 2 * H + GAP / 2]) - (e1 + e2) / 3
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    q *= np.sign(np.linalg.det(q))
    shift = rng.uniform(-0.5, 0.5, 3)
    place = lambda x: np.asarray(x) @ q.T + shift
    en = np.arange(1, 17, dtype=np.int32).reshape(2, 8)
    return rvf.MeshData(np.asfortranarray(place(p).T), en, np.zeros(2, dtype=np.int8), np.array([1, 2], dtype=np.int32),
                        {1: "lower", 2: "upper"}, {7: place([v0, v0 + e1, v0 + e2])[None]}, 2)


@pytest.mark.parametrize("cull", [True, False])
def test_tip_to_tip(rvf, orc, session, cull):
    from rvf_b200 import _abi
    wrong = []
    for seed in range(48):
        md = domes(rvf, seed)
        raw, area, _, _ = orc.solve_plain(orc.Mesh(md, [7]), 3, geometric=True)
        Fo = orc.f_from_raw(raw, area)[0, 1]
        raw, area, _, _ = orc.solve_plain(orc.Mesh(md, []), 3)
        open_ = orc.f_from_raw(raw, area)[0, 1]
        assert Fo < 1e-4 * open_, "the triangle must block the tips' ray"
        dm = _abi.DeviceMesh(session, rvf.mesh_desc_arrays(md, [7]))
        try:
            F = np.empty((2, 2), order="F")
            o = rvf.make_options(3, precision="mixed", geometric_soup=True, seed=0)
            o.disable_tile_cull = 0 if cull else 1
            dm.solve(o, F)
        finally:
            dm.release()
        if F[0, 1] > 1e-3 * open_:
            wrong.append((seed, F[0, 1], Fo))
    assert wrong == []
