"""floor_i64 and int_f64 (rusterize_gb300/csrc/rz_bits.h) against libm, on the
host, over edge values, halves, integers' neighbours and random bit patterns."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "rusterize_gb300" / "csrc"

CHECKER = r"""
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <cstring>
#include <random>
#include "rz_bits.h"

static int64_t ref_floor(double t) {
  if (std::isnan(t)) return 0;
  const double f = std::floor(t);
  const double lim = 4611686018427387904.0;  // 2^62
  if (f >= lim) return 1ll << 62;
  if (f <= -lim) return -(1ll << 62);
  return (int64_t)f;
}

int main() {
  long bad = 0;
  auto check = [&](double t) {
    if (rzb::floor_i64(t) != ref_floor(t)) { if (bad < 5) std::printf("floor %.17g\n", t); ++bad; }
  };
  auto conv = [&](int64_t n) {
    const double d = rzb::int_f64(n), r = (double)n;
    if (std::memcmp(&d, &r, 8)) { if (bad < 5) std::printf("int %lld\n", (long long)n); ++bad; }
  };
  const double sp[] = {0.0, -0.0, 0.5, -0.5, 1.0, -1.0, 5e-324, -5e-324, 0.9999999999999999, -0.9999999999999999,
                       4503599627370495.5, -4503599627370495.5, 4503599627370496.0, 9007199254740993.0, 1e18, -1e18,
                       4611686018427387904.0, -4611686018427387904.0, 1e300, -1e300, INFINITY, -INFINITY, NAN, -NAN};
  for (double t : sp) check(t);
  std::mt19937_64 rng(7);
  for (int i = 0; i < 3000000; ++i) {
    uint64_t b = rng();
    double t;
    switch (i % 4) {
      case 0: std::memcpy(&t, &b, 8); break;
      case 1: t = (double)(int64_t)(b % 4000000) / 7.0 - 200000.0; break;
      case 2: t = (double)(int64_t)(b % 100000) - 50000.5; break;
      default: t = std::nextafter((double)(int64_t)(b % 100000) - 50000.0, (i & 4) ? 1e9 : -1e9);
    }
    check(t);
    conv((int64_t)b >> (10 + i % 53));
  }
  for (int64_t n = -70000; n <= 70000; ++n) conv(n);
  conv(1ll << 53);
  conv(-(1ll << 53));
  conv((1ll << 53) - 1);
  std::printf("checked, %ld failures\n", bad);
  return bad != 0;
}
"""


def test_floor_and_conversion(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "c.cpp", tmp_path / "c"
    src.write_text(CHECKER)
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout[-2000:]
