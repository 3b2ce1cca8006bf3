"""Which caller's buffers a query kernel may use in place (span.h): all n ints
inside one page-locked range, aligned."""
import os
import subprocess

from conftest import REPO

MAIN = r"""
#include <cstdio>
#include "span.h"
int main() {
  const unsigned long long S = 65536, A = 1 << 20;
  struct { unsigned long long p; long long n; unsigned long long start, size; bool want; } t[] = {
      {A, 16384, A, S, true},                 // the whole range
      {A, 16385, A, S, false},                // runs on past it
      {A + 4, 16384, A, S, false},
      {A + 4, 16383, A, S, true},
      {A + S - 4, 1, A, S, true},
      {A + S, 1, A, S, false},                // starts behind it
      {A - 4, 2, A, S, false},                // starts before it
      {A + 2, 100, A, S, false},              // not aligned
      {A + 1, 1, A, S, false},
      {A, 16384, A, S - 1, false},            // a range that ends inside the last int
      {A, 1ll << 62, A, S, false},
      {A, 1, 0, 0, false},                    // no range known
      {A, 0, A, S, true},
  };
  int bad = 0, k = 0;
  for (auto &c : t) {
    if (gh::ints_inside(c.p, c.n, c.start, c.size) != c.want) { std::printf("case %d\n", k); bad = 1; }
    k++;
  }
  return bad;
}
"""


def test_ints_inside(tmp_path):
    src, exe = tmp_path / "span.cpp", str(tmp_path / "span")
    src.write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-I" + os.path.join(REPO, "gpu-h2h_gb300", "csrc"), str(src),
                           "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
