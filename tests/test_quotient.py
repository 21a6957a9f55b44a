"""The quotient of entry.cuh (a reciprocal and two fused corrections, Markstein 1990)
against IEEE division, bit for bit: the divisions of the Bessel recurrences, whole
numbers by R and recurrence values by whole numbers.  Runs the same operations on the
CPU (std::fma), where both roundings are IEEE's."""
import os
import subprocess

SRC = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>
static double quotient(double a, double b, double y) {
  double q = a * y;
  q = std::fma(std::fma(-b, q, a), y, q);
  return std::fma(std::fma(-b, q, a), y, q);
}
int main() {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  long bad = 0;
  for (long t = 0; t < 3000000; ++t) {
    // R over the accepted range (kQuotLo .. kQuotHi), the usual decades and neighbours of whole numbers
    double R = t % 4 == 0 ? std::pow(10.0, -20.0 + 40.0 * u(g)) : t % 4 == 1 ? 1.0 + 200.0 * u(g)
             : t % 4 == 2 ? std::nextafter((double)(1 + g() % 300), u(g) < 0.5 ? 0.0 : 1e9) : std::pow(10.0, -3.0 + 6.0 * u(g));
    const double rR = 1.0 / R;
    for (int k = 2; k <= 400; k += 2 + (int)(g() % 40)) bad += quotient(k, R, rR) != k / R;
    // recurrence values: 1e-250 .. 1e212, either sign
    const double x = (u(g) < 0.5 ? -1.0 : 1.0) * std::pow(10.0, -250.0 + 462.0 * u(g));
    const double kk = (double)(1 + g() % 1500);
    bad += quotient(x, kk, 1.0 / kk) != x / kk;
  }
  std::printf("%ld\n", bad);
}
"""


def test_quotient_is_correctly_rounded(tmp_path):
    c, e = tmp_path / "q.cpp", tmp_path / "q"
    c.write_text(SRC)
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-ffp-contract=off", str(c), "-o", str(e)])
    assert int(subprocess.check_output([str(e)], timeout=300)) == 0
