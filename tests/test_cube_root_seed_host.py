"""The Float64 cube root's seed (csrc/vf_exact.h) with a Float32 start that is as far off
as the hardware's is allowed to be, 2^-19 relative in either direction: within the
bound that its comment derives."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "volumefluxes.jl_gb300" / "csrc"

DRIVER = r"""
#include "vf_exact.h"
#include <cstdio>
#include <random>
using namespace vf::exact;
int main() {
  std::mt19937_64 g(11);
  double worst = 0;
  for (long i = 0; i < 2000000; ++i) {
    double t = from_bits((g() & 0xfffffffffffffull) | (1023 + g() % 3) << 52);
    if (i % 16 == 0) t = from_bits(bits((double)(1 << (i / 16 % 3))) + g() % 64);  // next to 1, 2, 4
    const long double r = std::cbrt((long double)t);
    worst = std::fmax(worst, (double)std::fabs(((long double)cube_root_seed(t) - r) / r) * 0x1p53);
  }
  std::printf("%g units of 2^-53\n", worst);
  return worst > 5.3;
}
"""


@pytest.mark.parametrize("error", ["0x1p-19", "-0x1p-19"])
def test_cube_root_seed_bound(tmp_path, error):
    src, exe = tmp_path / "driver.cpp", tmp_path / "driver"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-DVF_CBRT_SEED_ERROR={error}", f"-I{CSRC}",
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
