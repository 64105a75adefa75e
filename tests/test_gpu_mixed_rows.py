"""The packed FP32 rows of the quadrature-only kernel (fast_mixed_rows): for rules
of 1 to 64 points a block holds none, some or all of (odd and even blocks, whole and
remaining ones) and for partial tiles, F equals that of the generation kernel's
scalar operations, which an unclassified solve runs, bit for bit."""
import numpy as np
import pytest

from test_gpu_tile_cull import solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,nquad", [("tri3", 1), ("tri3", 2), ("quad4", 2), ("tri3", 3), ("quad4", 3), ("tri3", 4),
                                          ("quad4", 4), ("quad", 5), ("quad4", 7), ("quad4", 8)])
@pytest.mark.parametrize("m", [3, 6])
def test_rows(rvf, session, family, nquad, m):
    md = rvf.meshes.parallel_plates(m, family, gap=3.0)
    F, A, st = solve(rvf, session, md, nquad, [], precision="mixed")
    F0, A0, st0 = solve(rvf, session, md, nquad, [], precision="mixed", cull=False)
    assert np.array_equal(A, A0)
    assert np.array_equal(F, F0, equal_nan=True), f"max |dF| {np.nanmax(np.abs(F - F0))}"
    assert st["n_point_pairs"] == st0["n_point_pairs"]
