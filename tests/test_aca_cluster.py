"""The CTAs of an ACA job (csrc/aca_cluster.h): two, four or eight by the jobs of the level,
so that a level cut into launches of any size gives each of its jobs the same cluster,
and with it the same order of the sums that end its iteration."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aifmm_ls_b200", "csrc")
SRC = r"""
#include <cstdio>
#include <initializer_list>
#include "aca_cluster.h"
int main() {
  for (long boxes = 16; boxes <= 1 << 20; boxes *= 4) std::printf("%d ", aca_cluster_size(2 * boxes));
  for (long jobs : {1L, 296L, 297L, 592L, 593L}) std::printf("%d ", aca_cluster_size(jobs));
  std::printf("\n");
}
"""


def test_cluster_by_the_jobs_of_a_level(tmp_path):
    c, e = tmp_path / "a.cpp", tmp_path / "a"
    c.write_text(SRC)
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-I", CSRC, str(c), "-o", str(e)])
    got = [int(v) for v in subprocess.check_output([str(e)]).split()]
    # 32, 128, 512, 2,048 .. jobs, then around 2,368 CTAs
    assert got == [8, 8, 4, 2, 2, 2, 2, 2, 2] + [8, 8, 4, 4, 2]


def test_the_assembly_asks_with_the_level():
    with open(os.path.join(CSRC, "solver.cu")) as f:
        calls = re.findall(r"aifmm_launch_aca\(dj, nj, (.*?), tol", f.read())
    assert calls == ["2L * nbx"]  # both directions of every box, not the nj jobs of a chunk
