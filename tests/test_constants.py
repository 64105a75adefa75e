"""The constants that the CPU tests restate are the headers' (compiled for the host)."""
import subprocess

from conftest import load_pkg

PROGRAM = r"""
#include <cstdio>
#include "device_mixed.cuh"
int main() { std::printf("%.17g %.17g\n", (double)rvf::kMtTight.e0, (double)rvf::kMtTight.d); }
"""


def test_triangle_test_allowances(tmp_path):
    import test_mt_tolerance as t
    load_pkg()
    from rvf_b200 import build
    (tmp_path / "c.cu").write_text(PROGRAM)
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-o", str(tmp_path / "c"), str(tmp_path / "c.cu")], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([str(tmp_path / "c")], check=True, capture_output=True, text=True).stdout
    assert tuple(map(float, out.split())) == (t.E0, t.D)
