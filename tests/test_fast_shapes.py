"""Which quadrature-only kernel a solve runs (fast_flat, kernels.h, compiled for the
host): a point block that the caller names is the one that runs."""
import subprocess

from conftest import load_pkg

PROGRAM = r"""
#include <cstdio>
#include "kernels.h"
int main() {
  for (int mixed = 0; mixed < 2; ++mixed)
    for (int dim3 = 0; dim3 < 2; ++dim3)
      for (int pmax : {1, 3, 4, 7, 9, 64})
        for (int groups : {1, 2, 4, 8, 32})
          for (int qb : {0, 2, 3, 4})
            std::printf("%d %d %d %d %d %d\n", mixed, dim3, pmax, groups, qb,
                        (int)rvf::fast_flat(mixed != 0, dim3 != 0, pmax, groups, qb));
}
"""


def test_row_set_kernel_only_by_the_rule(tmp_path):
    load_pkg()
    from rvf_b200 import build
    (tmp_path / "f.cu").write_text(PROGRAM)
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-o", str(tmp_path / "f"), str(tmp_path / "f.cu")], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([str(tmp_path / "f")], check=True, capture_output=True, text=True).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(rows) == 2 * 2 * 6 * 5 * 4
    for mixed, dim3, pmax, groups, qb, flat in rows:
        assert flat == (not mixed and dim3 and pmax <= 7 and groups <= 8 and qb == 0)
