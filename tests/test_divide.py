"""The division of cell and row indices by the grid edge as a multiplication
(csrc/ggb_divide.h), compiled and run on the host: exact for every index around
the multiples of N where a quotient changes, for edges up to the largest that
cs_init takes."""
import os
import subprocess

from conftest import PKG

PROBE = r"""
#include <cstdio>
#include "ggb_divide.h"
using namespace ggb;
static long bad = 0, tried = 0;
static void check(int N) {
  const unsigned long long f = div_factor(N);
  const long n = 6L * N * N;
  auto one = [&](long c) {
    if (c < 0 || c >= n) return;
    tried++;
    if (div_by((unsigned)c, f) != (int)(c / N)) bad++;
  };
  // rows: every one of a small grid, else the first, the last and every 97th
  for (long r = 0; r <= 6L * N; r += (N < 600 || r < 4 || r > 6L * N - 100) ? 1 : 97)
    for (int d = -1; d <= 1; d++) one(r * N + d);
  for (int r = 0; r < 6 * N; r++) {
    tried++;
    if (div_by((unsigned)r, f) != r / N) bad++;
  }
}
int main() {
  for (int N = 1; N <= 16384; N++) check(N);
  printf("%ld %ld\n", bad, tried);
}
"""


def test_division_is_exact(tmp_path):
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text(PROBE)
    subprocess.run(["/usr/bin/g++", "-O2", "-std=c++17", f"-I{os.path.join(PKG, 'csrc')}", "-o", str(exe), str(src)],
                   check=True)
    bad, tried = map(int, subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert tried > 10**8 and bad == 0
