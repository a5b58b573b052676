"""st3d_f64.cuh compiled for the CPU: every sum that the integer path serves is
the double sum bit for bit, no operation in it is undefined for any operand
(the undefined-behaviour sanitizer ends the program), and the range check keeps
infinities, NaN, zeros and subnormals out."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stencil3d_gb300", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <vector>
#include "st3d_f64.cuh"
using namespace st3d;
static uint64_t state = 88172645463325252ull;
static uint64_t draw() { state ^= state << 13; state ^= state >> 7; state ^= state << 17; return state; }
static double make(uint64_t exponent) {
  const uint64_t b = (draw() & 0x800fffffffffffffull) | ((exponent > 2047 ? 2047 : exponent) << 52);
  double x;
  memcpy(&x, &b, 8);
  return x;
}
static long served = 0, wrong = 0;
static void pair(double a, double b, double u) {
  const Twice t = twice_of(u);
  uint32_t E;
  double d;
  if (!pair_fits(bits_of(a), bits_of(b), t, &E)) return;
  if (!pair_diff_bits(bits_of(a), bits_of(b), t, E, &d)) return;
  const double want = (a + b) - (u + u);
  ++served;
  wrong += memcmp(&want, &d, 8) != 0 || !std::isfinite(a) || !std::isfinite(b) || !std::isfinite(u);
}
int main() {
  const double inf = INFINITY;
  std::vector<double> ends = {0.0, -0.0, 5e-324, -2e-308, inf, -inf, std::nan(""), 1.7e308, -8.9e307, 9e307, 1.0};
  for (double a : ends)
    for (double b : ends)
      for (double u : ends) pair(a, b, u);
  for (long n = 0; n < 2000000; ++n) {
    const uint64_t e = draw() % 2048;
    const double a = make(e + draw() % 12), b = make(e + draw() % 12), u = make(n % 8 ? e + draw() % 12 : draw() % 2048);
    pair(a, b, u);
  }
  printf("%ld %ld\n", served, wrong);
  return 0;
}
"""


def test_integer_sums_are_defined_and_exact(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "sums.cpp", tmp_path / "sums"
    src.write_text(PROGRAM)
    cmd = ["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-x", "c++", str(src), "-o", str(exe)]
    checked = cmd[:1] + ["-fsanitize=undefined", "-fno-sanitize-recover=undefined"] + cmd[1:]
    if subprocess.run(checked, capture_output=True).returncode != 0:
        subprocess.run(cmd, check=True)  # no sanitizer library: the sums alone
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    served, wrong = map(int, r.stdout.split())
    assert served > 500000 and wrong == 0
