"""Scratch sizes of a service batch (csrc/pwa_scratch.h): batches of few large
fits and of many small ones in turn settle on sizes that hold both, so nothing
is allocated after the first of each."""
import itertools
import os
import subprocess

from common import ROOT

# (counters, argument bytes, rows of 5 sums): two fits of 16384 tiles, 300
# fits of one tile, 40 of 1024, at two columns
BATCHES = [(259, 168, 42_240), (601, 21_624, 7_500), (681, 2_904, 207_200)]

HARNESS = """
#include <cstdio>
#include "pwa_scratch.h"
int main() {
  BatchScratch s;
  long long c, a, r;
  while (std::scanf("%lld %lld %lld", &c, &a, &r) == 3) {
    const bool kept = s.holds(c, (size_t)a, r);
    const BatchScratch g = kept ? s : s.grown(c, (size_t)a, r);
    if (!g.holds(c, (size_t)a, r) || g.counters < s.counters || g.args < s.args ||
        g.rows < s.rows || (sizeof(unsigned int) * g.counters) % 256 || g.args % 256 ||
        g.bytes() != sizeof(unsigned int) * g.counters + g.args + sizeof(double) * g.rows)
      return 1;
    s = g;
    std::printf("%d\\n", kept ? 0 : 1);
  }
  return 0;
}
"""


def test_alternating_batches(tmp_path):
    src, exe = tmp_path / "scratch.cpp", tmp_path / "scratch"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "tf-pwa_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    for order in itertools.permutations(BATCHES):
        text = "\n".join(" ".join(map(str, b)) for b in order * 4)
        r = subprocess.run([str(exe)], input=text, capture_output=True, text=True)
        assert r.returncode == 0, order
        allocated = [int(x) for x in r.stdout.split()]
        assert allocated[0] == 1 and not any(allocated[len(order):]), (order, allocated)
