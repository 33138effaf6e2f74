"""all_touched segments walked in fixed point (rusterize_gb300/csrc/rz_bits.h
touch_dda) against the reference's FP64 walk on the host: every pixel in order
up to where the fixed-point walk gives a decision back, over slopes, sizes,
integer end points and points near pixel corners; and the kernel, which then
continues in FP64, against the oracle."""

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from rusterize_gb300 import geometry as G

from _util import diff_report, gpu_burn, oracle_burn, same_bits

CSRC = Path(__file__).resolve().parents[1] / "rusterize_gb300" / "csrc"

CHECKER = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <utility>
#include "rz_bits.h"

int main() {
  std::mt19937_64 rng(3);
  auto uni = [&](double a, double b) { return a + (b - a) * (double)(rng() >> 11) * 0x1p-53; };
  const int sizes[][2] = {{40, 30}, {1500, 2500}, {70000, 300}, {300, 70000}, {4000000, 4000000}, {1, 1}, {3, 2}};
  long bad = 0, walks = 0, whole = 0, pixels = 0;
  for (int it = 0; it < 800000; ++it) {
    const int ncols = sizes[it % 7][0], nrows = sizes[it % 7][1];
    double x = uni(-3, ncols + 3), y = uni(-3, nrows + 3);
    const double len = std::exp2(uni(-6, 9));
    double xe = x + len * uni(-1, 1), ye = y + len * uni(-1, 1);
    switch ((it / 7) % 8) {
      case 0: x = std::floor(x); y = std::floor(y); break;
      case 1: xe = std::floor(xe); ye = std::floor(ye); break;
      case 2: ye = std::floor(ye) + std::exp2(-uni(10, 60)); break;
      case 3: xe = std::floor(xe) - std::exp2(-uni(10, 60)); break;
      case 4: {  // through (nearly) a pixel corner
        const double cx = std::floor(uni(x, xe)) - x, cy = std::floor(uni(y, ye)) - y + std::exp2(-uni(10, 60));
        const double k = uni(1, 3);
        xe = x + k * cx;
        ye = y + k * cy;
        break;
      }
      case 5: ye = y + (ye - y) * std::exp2(-uni(0, 12)); break;
      case 6: xe = x + (xe - x) * std::exp2(-uni(0, 12)); break;
      default: break;
    }
    if (x > xe) { std::swap(x, xe); std::swap(y, ye); }
    if (std::fabs(x - xe) < 0.01 || std::fabs(y - ye) < 0.01) continue;
    const double s = (ye - y) / (xe - x), inv = 1.0 / s;
    if (x < 0) { y += (0 - x) * s; x = 0; }
    if (xe > ncols) { ye += (ncols - xe) * s; xe = ncols; }
    if (y < 0) { x += (0 - y) * inv; y = 0; } else if (y > nrows) { x += (nrows - y) * inv; y = nrows; }
    if (ye < 0) xe += (0 - ye) * inv; else if (ye > nrows) xe += (nrows - ye) * inv;
    x = std::fmin(std::fmax(x, 0.0), (double)ncols);
    xe = std::fmin(std::fmax(xe, 0.0), (double)ncols);
    if (!(x < xe)) continue;
    rzb::TouchDda w;
    if (!rzb::touch_dda(x, y, xe, s, inv, ncols, nrows, w)) continue;
    ++walks;
    bool ok = true, edge = false, more = true;
    while (true) {
      const long long ix = (long long)std::floor(x), iy = (long long)std::floor(y);
      ++pixels;
      if (ix != w.ix || iy != w.iy + (edge ? 1 : 0)) { ok = false; break; }
      // the FP64 step
      const double tol = 1e-9;
      double sx = std::floor(x + 1.0) - x, sy = sx * s;
      if ((long long)std::floor(y + sy) == iy) {
        x += sx;
        y += sy;
      } else if (s < 0) {
        sy = (double)iy - y;
        if (sy > -tol) sy = -tol;
        sx = sy / s;
        x += sx;
        y += sy;
      } else {
        sy = (double)(iy + 1) - y;
        if (sy < tol) sy = tol;
        sx = sy / s;
        x += sx;
        y += sy;
      }
      const bool on = x >= 0 && x < xe;
      if (edge) {
        edge = false;
        if (!on) { ok = false; break; }
        continue;
      }
      bool row;
      const int r = rzb::touch_step(w.g, w.a, w.b, w.a_last, w.ix, w.end, w.iy, w.margin, w.up, row);
      if (r == rzb::TOUCH_UNSURE) break;
      more = r == rzb::TOUCH_NEXT;
      if (more != on) { ok = false; break; }
      if (!more) { ++whole; break; }
      edge = row && w.up;
    }
    if (!ok && ++bad < 6) std::printf("walk %d: %d x %d, slope %.17g\n", it, ncols, nrows, s);
  }
  std::printf("%ld walks, %ld to their end, %ld pixels, %ld failures\n", walks, whole, pixels, bad);
  return bad != 0 || whole < walks / 2 || walks < 200000;
}
"""


def test_fixed_point_walk(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src = tmp_path / "c.cpp"
    src.write_text(CHECKER)
    exe = tmp_path / "c"
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("grain", [0.0, 1.0, 0.125])
def test_walks_that_change_to_fp64(grain):
    # grain 1: vertices on pixel corners; 0.125: segments through corners at their middle
    rng = np.random.default_rng(int(8 * grain))
    b = G.TableBuilder()
    for k in range(60):
        n = int(rng.integers(2, 40))
        xy = np.cumsum(np.vstack([rng.uniform(-5, 205, (1, 2)), rng.normal(0, 2.0 ** (k % 8), (n, 2))]), axis=0)
        if grain:
            xy = np.round(xy / grain) * grain + (0.5 - 2.0 ** -40 if k % 3 == 0 else 0.0)
        G.add_linestring(b, xy)
    t = b.build()
    grid = dict(nrows=190, ncols=201, xmin=0.0, xmax=201.0, ymin=0.0, ymax=190.0, xres=1.0, yres=1.0)
    for fn, dt in (("sum", "float32"), ("last", "int16"), ("count", "uint8")):
        kw = dict(fn=fn, values=np.arange(1, t.n_geoms + 1).astype(dt), background=0, dtype=dt, all_touched=True)
        got, ref = gpu_burn(t, grid, **kw), oracle_burn(t, grid, **kw)
        assert same_bits(got, ref), f"{fn}: " + diff_report(got, ref)
