"""The integer forms of Float64 operations (csrc/vf_exact.h) against the CPU's
IEEE division, square root and products, bit for bit: random bit patterns,
significands of all ones, nearly all ones, few bits and shifted runs, operands
a few ulps apart (quotients next to 1), squares moved by a few ulps (roots next
to representable numbers), subnormals, zeros and infinities; with the Float32
seeds moved by an ulp in either direction, as the hardware's may be."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "volumefluxes.jl_gb300" / "csrc"

DRIVER = r"""
#include "vf_exact.h"
#include <cstdio>
#include <random>
using namespace vf::exact;
static long bad = 0;
static void same(const char* what, double x, double y, double got, double want) {
  if (bits(got) == bits(want) || (got != got && want != want)) return;
  if (bad++ < 5) std::printf("%s %a %a: %a, want %a\n", what, x, y, got, want);
}
int main() {
  std::mt19937_64 g(7);
  auto any = [&] { return from_bits(g()); };
  auto shaped = [&] {
    const u64 all = 0xfffffffffffffull, r = g();
    u64 m = r & all;
    switch (g() % 7) {
      case 0: m = 0; break;
      case 1: m = all; break;
      case 2: m &= g() & g() & g(); break;
      case 3: m = (m | g() | g() | g()) & all; break;
      case 4: m >>= g() % 52; break;
      case 5: m = (m >> (g() % 52)) ^ all; break;
    }
    return from_bits(m | (1020 + g() % 7) << 52 | (g() & 1) << 63);
  };
  for (long i = 0; i < COUNT; ++i) {
    double a = i % 4 ? shaped() : any(), b = i % 4 ? shaped() : any();
    if (i % 16 == 1) b = from_bits(bits(a) + g() % 64 - 32);
    if (i % 16 == 3) a = from_bits(bits(a) & 0x801fffffffffffffull);  // subnormal or the smallest normal binades
    same("quotient", a, b, quotient(divisor(b), a), a / b);
    same("half", a, 0, half(a), 0.5 * a);
    same("zero_minus", a, 0, zero_minus(a), [](volatile double z, double v) { return z - v; }(0.0, a));
    const int k = (int)(g() % 40) - 20;
    same("scale_pow2", a, k, scale_pow2(a, k, std::ldexp(1.0, k)), a * std::ldexp(1.0, k));
    double x = std::fabs(a);
    if (i % 8 == 5) x = from_bits(bits(x * x) + g() % 8 - 4);
    same("square_root", x, 0, square_root(x), std::sqrt(x));
  }
  const double special[] = {0.0, -0.0, HUGE_VAL, -HUGE_VAL, 1.0, -1.0, 4.9e-324, 2.2250738585072014e-308, 1.7976931348623157e308};
  for (double a : special) {
    same("square_root", a, 0, square_root(a), std::sqrt(a));
    same("half", a, 0, half(a), 0.5 * a);
    for (double b : special) same("quotient", a, b, quotient(divisor(b), a), a / b);
  }
  double worst = 0;
  for (long i = 0; i < COUNT / 8; ++i) {
    const double t = from_bits((g() & 0xfffffffffffffull) | (1023 + g() % 3) << 52);
    const long double r = std::cbrt((long double)t);
    worst = std::fmax(worst, (double)std::fabs((long double)cube_root_seed(t) - r) * 0x1p52);
  }
  if (worst > 4) { std::printf("cube_root_seed is %g ulps off\n", worst); ++bad; }
  return bad != 0;
}
"""


@pytest.mark.parametrize("seed_ulps", [0, 1, -1])
def test_integer_forms_equal_ieee(tmp_path, seed_ulps):
    cxx = shutil.which("g++")
    assert cxx, "g++ is part of the toolchain"
    src, exe = tmp_path / "driver.cpp", tmp_path / "driver"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", f"-DVF_SEED_ULPS={seed_ulps}", "-DCOUNT=4000000L",
                    f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
