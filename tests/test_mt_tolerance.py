"""The tight allowances of the FP32 triangle test (kMtTight, device_mixed.cuh):
the numerators formed in FP32, with every input rounded as the kernels round it,
stay within half of the allowed distance from their exact values (the bounds
derived there leave a factor two)."""
import numpy as np
import pytest

E0, D = 3.814697265625e-06, 1.25
f32 = np.float32


def fma(a, b, c):
    """float32 fma: the product is exact in float64, the sum rounded twice."""
    return f32(np.float64(a) * np.float64(b) + np.float64(c))


def cross(a, b):
    return [fma(a[1], b[2], -f32(a[2] * b[1])), fma(a[2], b[0], -f32(a[0] * b[2])), fma(a[0], b[1], -f32(a[1] * b[0]))]


def dot(a, b):
    return fma(a[0], b[0], fma(a[1], b[1], f32(a[2] * b[2])))


@pytest.mark.parametrize("from_centroids", [False, True])
@pytest.mark.parametrize("seed", range(3))
def test_numerators(seed, from_centroids):
    rng = np.random.default_rng(seed)
    n = 200_000
    mx = 10.0 ** rng.uniform(-2, 2)  # largest coordinate
    extent = 1.0 + mx
    ci, cj = rng.uniform(-mx, mx, (2, 3, n)) * 0.8
    # elements of at most half the centroid distance, points within 0.6 diameters
    diam = 0.5 * np.linalg.norm(cj - ci, axis=0) * rng.uniform(0.01, 1.0, n)
    diam = np.minimum(diam, 0.15 * mx)
    op, oq = (rng.normal(size=(2, 3, n)) / 3.0).clip(-0.34, 0.34) * diam
    o, r = ci + op, (cj + oq) - (ci + op)
    # triangles around a point of the ray
    at = o + rng.uniform(0, 1, n) * r
    size = mx * 10.0 ** rng.uniform(-3, -0.5, n)
    v0, v1, v2 = (at + rng.normal(size=(3, n)) * size for _ in range(3))
    v0, v1, v2 = (v.clip(-mx, mx) for v in (v0, v1, v2))
    e1, e2 = v1 - v0, v2 - v0
    # as the kernels round
    if from_centroids:
        p32, q32, d32 = f32(op), f32(oq), f32(cj - ci)
        r32 = d32 + (q32 - p32)
        o32 = f32(ci) + p32
    else:
        r32, o32 = f32(r), f32(o)
    r2 = fma(r32[0], r32[0], fma(r32[1], r32[1], f32(r32[2] * r32[2])))
    inv = f32(1.0 / np.sqrt(np.float64(r2))) * f32(1.0 + 2.0 ** -22)  # rsqrt within two units
    d = [c * inv for c in r32]
    E1, E2, V0 = f32(e1), f32(e2), f32(v0)
    s = [o32[k] - V0[k] for k in range(3)]
    h, q = cross(d, E2), cross(s, E1)
    U, V, T, a = dot(s, h), dot(d, q), dot(E2, q), dot(E1, h)
    # exact
    dx = r / np.linalg.norm(r, axis=0)
    sx = o - v0
    hx, qx = np.cross(dx.T, e2.T).T, np.cross(sx.T, e1.T).T
    n1, n2 = np.linalg.norm(e1, axis=0), np.linalg.norm(e2, axis=0)
    ns, d2 = np.abs(sx).sum(axis=0), D * 2.0 ** -20 * extent
    e = E0 * (ns + d2) + d2
    for got, want, bound in ((U, (sx * hx).sum(0), e * n2), (V, (dx * qx).sum(0), (e + d2) * n1),
                             (T, (e2 * qx).sum(0), (e + d2) * n1 * n2), (a, (e1 * hx).sum(0), E0 * n1 * n2)):
        assert (np.abs(np.float64(got) - want) / bound).max() < 0.5
