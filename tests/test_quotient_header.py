"""quotient() as the entries include it (csrc/quotient.cuh) against IEEE division, bit for
bit, compiled for the host and for the device: whole numbers by R over the accepted
range (kQuotLo .. kQuotHi) and recurrence values by whole numbers."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aifmm_ls_b200", "csrc")
SRC = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "quotient.cuh"
struct Pair { double a, b; };
#ifdef __CUDACC__
__global__ void run(const Pair* p, double* q, double* d, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  q[t] = quotient(p[t].a, p[t].b, 1.0 / p[t].b);
  d[t] = p[t].a / p[t].b;
}
#endif
int main() {
  std::mt19937_64 g(9);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  std::vector<Pair> v;
  for (int t = 0; t < 1000000; ++t) {
    const double R = t % 3 == 0 ? kQuotLo * std::pow(kQuotHi / kQuotLo, u(g)) : t % 3 == 1 ? 1.0 + 200.0 * u(g)
                   : std::nextafter((double)(1 + g() % 300), u(g) < 0.5 ? 0.0 : 1e9);
    if (R > kQuotLo && R < kQuotHi) v.push_back({2.0 * (double)(1 + g() % 400), R});
    v.push_back({(u(g) < 0.5 ? -1.0 : 1.0) * std::pow(10.0, -250.0 + 462.0 * u(g)), (double)(1 + g() % 1500)});
  }
  const int n = (int)v.size();
  std::vector<double> q(n), d(n);
#ifdef __CUDACC__
  Pair* dp;
  double *dq, *dd;
  if (cudaMalloc(&dp, sizeof(Pair) * n) || cudaMalloc(&dq, 8 * n) || cudaMalloc(&dd, 8 * n)) return 1;
  cudaMemcpy(dp, v.data(), sizeof(Pair) * n, cudaMemcpyHostToDevice);
  run<<<(n + 255) / 256, 256>>>(dp, dq, dd, n);
  cudaMemcpy(q.data(), dq, 8 * n, cudaMemcpyDeviceToHost);
  if (cudaMemcpy(d.data(), dd, 8 * n, cudaMemcpyDeviceToHost)) return 1;
#else
  for (int t = 0; t < n; ++t) { q[t] = quotient(v[t].a, v[t].b, 1.0 / v[t].b); d[t] = v[t].a / v[t].b; }
#endif
  long bad = 0;
  for (int t = 0; t < n; ++t) bad += q[t] != v[t].a / v[t].b || d[t] != q[t];
  std::printf("%d %ld\n", n, bad);
}
"""


def _run(tmp_path, name, cmd):
    c, e = tmp_path / name, tmp_path / "q"
    c.write_text(SRC)
    subprocess.check_call(cmd + ["-O2", "-std=c++17", "-I", CSRC, str(c), "-o", str(e)])
    n, bad = (int(t) for t in subprocess.check_output([str(e)], timeout=300).split())
    assert n > 1500000 and bad == 0


def test_on_the_host(tmp_path):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    _run(tmp_path, "q.cpp", [cxx, "-ffp-contract=off"])


@pytest.mark.gpu
def test_on_the_device(tmp_path):
    from aifmm_ls_b200.build import ARCH, nvcc
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    _run(tmp_path, "q.cu", [nvcc()] + ARCH + ["-ccbin", cxx, "-Xcompiler", "-ffp-contract=off"])
