"""pow_two_thirds of the FP64 hexahedra against the host's long double power. The
header's function is compiled for the host with the device's names for the bits
of a double; the FP32 inverse cube root is the exact one moved by up to two units
in its last place, the device function's bound.

Bar: 2.2e-16 relative (one unit in the last place of a result just above a power
of two): the function it stands for, pow, is allowed as much."""
import shutil
import subprocess

import pytest

from weldformfem_gb300 import build as B

SRC = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#define __device__
#define __forceinline__ inline
static int g_ulp;
static uint64_t bits(double v) { uint64_t u; std::memcpy(&u, &v, 8); return u; }
static double from_bits(uint64_t u) { double v; std::memcpy(&v, &u, 8); return v; }
static int __double2hiint(double v) { return (int)(bits(v) >> 32); }
static int __double2loint(double v) { return (int)bits(v); }
static double __hiloint2double(int h, int l) {
  return from_bits(((uint64_t)(uint32_t)h << 32) | (uint32_t)l);
}
static float rcbrtf(float v) {
  float r = (float)(1.0 / std::cbrt((double)v));
  for (int i = 0; i < (g_ulp < 0 ? -g_ulp : g_ulp); i++) r = std::nextafterf(r, g_ulp < 0 ? 0.f : 1e38f);
  return r;
}
using std::fma; using std::pow;
#include "wf_hex.cuh"
int main() {
  uint64_t s = 88172645463325252ull;
  long double worst = 0;
  for (int i = 0; i < 600000; i++) {
    s ^= s << 13; s ^= s >> 7; s ^= s << 17;
    // volumes of 1e-15 to 1e-3 mostly, the whole range of the fast form, and
    // mantissas around the logarithm's cut
    const double u = (double)(s >> 11) * 0x1p-53;
    double v = i % 3 == 0 ? std::pow(10.0, -29.9 + 59.8 * u) : std::pow(10.0, -15.0 + 12.0 * u);
    if (i % 3 == 1) v = std::ldexp(1.4142 + 2e-4 * (u - 0.5), i % 80 - 50);
    g_ulp = i % 5 - 2;
    const long double want = powl((long double)v, (long double)0.6666666);
    const long double e = fabsl((long double)wf::pow_two_thirds(v) / want - 1.0L);
    if (e > worst) worst = e;
  }
  std::printf("%.3Le\n", worst);
  for (double v : {0.0, 1e-31, 3e30, -1.0})
    if (bits(wf::pow_two_thirds(v)) != bits(std::pow(v, 0.6666666)) && v >= 0) return 1;
  return std::isnan(wf::pow_two_thirds(-1.0)) ? 0 : 1;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_power_is_as_accurate_as_pow(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", B.CSRC,
                    str(tmp_path / "t.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, check=True)
    assert float(r.stdout) <= 2.2e-16, r.stdout
