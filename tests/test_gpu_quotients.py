"""Quotients by one divisor (div_by, div_all, device_common.cuh) on the device,
bit for bit the division's for every numerator and positive divisor that
div_by_ok lets through: signs of zero, the ends of its range, and numerators and
divisors at opposite ends of it."""
import subprocess

import pytest

from conftest import load_pkg

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "device_common.cuh"
using namespace rvf;

__global__ void k(int n, const double* a, const double* b, unsigned long long* bad, unsigned long long* taken) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double q = a[i] / b[i];
  if (div_by_ok(a[i]) && div_by_ok(b[i])) {
    atomicAdd(taken, 1ull);
    if (__double_as_longlong(div_by(a[i], b[i], 1.0 / b[i])) != __double_as_longlong(q)) atomicAdd(bad, 1ull);
  }
  const double v[2] = {a[i], -a[i]};
  double r[2];
  div_all(v, b[i], r);
  if (__double_as_longlong(r[0]) != __double_as_longlong(q) || __double_as_longlong(r[1]) != __double_as_longlong(-q))
    atomicAdd(bad + 1, 1ull);
}

int main() {
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> U(1.0, 2.0);
  std::uniform_int_distribution<int> wide(-705, 705), narrow(-40, 40);
  const double ends[] = {1.0, 1.0 + 0x1p-52, 2.0 - 0x1p-52, 1.5, 4.0 / 3.0};
  const int exps[] = {-1074, -1022, -701, -700, -699, -501, -500, -499, -1, 0, 1, 498, 499, 500, 698, 699, 700, 1023};
  std::vector<double> a, b;
  auto add = [&](double x, double y) { a.push_back(x), b.push_back(y); };
  for (int k = 0; k < 1 << 20; ++k) {
    add(std::ldexp(U(g), wide(g)) * (k & 1 ? -1 : 1), std::ldexp(U(g), wide(g)));
    add(std::ldexp(U(g), narrow(g)) * (k & 1 ? -1 : 1), std::ldexp(U(g), narrow(g)));
  }
  for (double m : ends)
    for (double n : ends)
      for (int e : exps)
        for (int f : exps) add(std::ldexp(m, e), std::ldexp(n, f)), add(-std::ldexp(m, e), std::ldexp(n, f));
  for (int f : exps) add(0.0, std::ldexp(1.5, f)), add(-0.0, std::ldexp(1.5, f));
  const int n = (int)a.size();
  double *da, *db;
  unsigned long long *d, h[3] = {0, 0, 0};
  if (cudaMalloc(&da, 8 * (size_t)n) || cudaMalloc(&db, 8 * (size_t)n) || cudaMalloc(&d, 24)) return 1;
  cudaMemcpy(da, a.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
  cudaMemset(d, 0, 24);
  k<<<(n + 255) / 256, 256>>>(n, da, db, d, d + 2);
  if (cudaMemcpy(h, d, 24, cudaMemcpyDeviceToHost)) return 1;
  std::printf("%llu %llu %llu\n", h[0], h[1], h[2]);
  return 0;
}
"""


def test_rounded_as_the_division(tmp_path):
    load_pkg()
    from rvf_b200 import build
    (tmp_path / "q.cu").write_text(PROGRAM)
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-o", str(tmp_path / "q"), str(tmp_path / "q.cu")], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([str(tmp_path / "q")], check=True, capture_output=True, text=True).stdout
    bad, bad_all, taken = map(int, out.split())
    assert taken > 1 << 20
    assert (bad, bad_all) == (0, 0)
