"""Band width of the near-far searches (csrc/gg_band.h) compiled for the host, with the
undefined-behaviour checks on: mean weights whose multiple leaves the distance type."""
import os
import subprocess

from conftest import PKG

PROGRAM = r"""
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <limits>
#include "gg_band.h"
template <typename T> static int check() {
  const double top = (double)std::numeric_limits<T>::max();
  int bad = 0;
  const double wants[] = {-1.0, 0.0, 0.3, 1.0, 31.5, 1e8 * 32, 6.8e7 * 32, 1e18 * 32, 1e39, 1e308, INFINITY, NAN};
  for (double w : wants) {
    const T d = gg::band_width<T>(w);
    if (!(d > T(0)) || (double)d > top / 4) ++bad;
    if (w >= top / 4 && (double)d < top / 8) ++bad;  // a wide band stays wide
    if (w >= 1.0 && w < top / 4 && (double)d != (double)(T)w) ++bad;
  }
  return bad;
}
int main() {
  const int bad = check<int32_t>() + check<int64_t>() + check<float>() + check<double>();
  printf("%d\n", bad);
  return bad != 0;
}
"""


def test_band_width_stays_in_the_type(tmp_path):
    src, exe = tmp_path / "band.cpp", tmp_path / "band"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined,float-cast-overflow",
                    "-fno-sanitize-recover=all", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
