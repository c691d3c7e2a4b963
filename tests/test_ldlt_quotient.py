"""The LDL^T panel's division by a reciprocal known ahead (ldlt_panel.cuh, quotient), compiled for the
host with the compiler's fused multiply-add: the bits of x / d over the whole range of exponents it
takes, at significands next to a power of two on both sides (all ones included), with trailing zeros
(exact quotients), and where it must take the division itself."""
import subprocess

from native import emulation as E

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include <random>
#include "cuda/ldlt_panel.cuh"
using namespace fc::ldlt;
int main() {
  std::mt19937_64 g(1);
  auto number = [&](int most, int kind) {
    uint64_t m = g() & 0xfffffffffffffull;
    if (kind == 1) m = 0xfffffffffffffull - (g() & 15);
    if (kind == 2) m = g() & 15;
    if (kind == 3) m &= ~0xffffffull;
    const uint64_t b = (g() & 1) << 63 | (1023 - most + g() % (2 * most + 1)) << 52 | m;
    double x;
    std::memcpy(&x, &b, 8);
    return x;
  };
  auto same = [](double x, double d) {
    const double a = x / d, b = quotient(x, d, reciprocal(d));
    return std::memcmp(&a, &b, 8) == 0 || (a != a && b != b);
  };
  for (int i = 0; i < 4000000; ++i) {
    const double x = number(i & 16 ? 620 : 3, i % 4), d = number(i & 16 ? 310 : 3, i / 4 % 4);
    if (!same(x, d)) return std::printf("%a / %a\n", x, d), 1;
  }
  const double inf = HUGE_VAL, nan = inf - inf;
  const double xs[] = {0.0, -0.0, inf, -inf, nan, 5e-324, -1e-310, 1.7e308, 1.0};
  for (double x : xs)
    for (double d : xs)
      if (!same(x, d)) return std::printf("%a / %a\n", x, d), 1;
  return 0;
}
"""


def test_every_quotient_is_the_divisions(tmp_path):
    src, exe = tmp_path / "quotient.cpp", tmp_path / "quotient"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{E.HEADER.parent.parent}", "-o", str(exe),
                    str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
