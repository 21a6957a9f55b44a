"""The opt-in to large dynamic shared memory (csrc/smem_limit.h): once for every device, not
once a process; not kept after an error; the same from many threads; devices beyond the
table are asked every time."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aifmm_ls_b200", "csrc")
SRC = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "smem_limit.h"
static SmemLimit limits[2];
int main() {
  int calls[100] = {0};
  bool fail = true;
  auto ask = [&](SmemLimit& l, int dev) { return l.once(dev, [&] { ++calls[dev < 0 ? 99 : dev]; return fail ? 7 : 0; }); };
  auto show = [&](SmemLimit& l, int dev) { std::printf("%d ", ask(l, dev)); };
  show(limits[0], 0); show(limits[0], 0);  // errors are returned and not kept
  fail = false;
  show(limits[0], 0); show(limits[0], 0); std::printf("%d ", calls[0]);
  show(limits[0], 1); show(limits[0], 1); std::printf("%d ", calls[1]);  // another device
  show(limits[1], 1); std::printf("%d ", calls[1]);                     // another kernel
  ask(limits[0], 64); ask(limits[0], 64); ask(limits[0], -1);
  std::printf("%d %d ", calls[64], calls[99]);
  static SmemLimit shared;
  std::atomic<int> raised{0}, wrong{0};
  std::vector<std::thread> ts;
  for (int t = 0; t < 16; ++t)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 20000; ++i)
        wrong += shared.once((t + i) % 8, [&] { ++raised; return 0; }) != 0;
    });
  for (auto& t : ts) t.join();
  const int before = raised;
  for (int d = 0; d < 8; ++d) shared.once(d, [&] { ++raised; return 0; });
  std::printf("%d %d %d\n", before >= 8 && before <= 128, (int)raised - before, (int)wrong);
}
"""


def test_limit_is_raised_once_for_each_device(tmp_path):
    c, e = tmp_path / "l.cpp", tmp_path / "l"
    c.write_text(SRC)
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-pthread", "-I", CSRC, str(c), "-o", str(e)])
    got = subprocess.check_output([str(e)], timeout=300).split()
    assert [int(v) for v in got] == [7, 7, 0, 0, 3, 0, 0, 1, 0, 2, 2, 1, 1, 0, 0]

