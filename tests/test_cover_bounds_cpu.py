"""The coverage test of the raster pass at the edge of k_emit's area rule, its
source compiled for the host: a listed triangle's area bound is computed once
more there, in another order of roundings, and may come out on the other side
of the area.  Such a triangle decides nothing: no point of it is called
certainly outside, none beyond it certainly inside.  Triangles of 2 to 100
bounds across, their third vertex moved to where the area meets its bound."""
import os
import subprocess

from contour3d_gb300 import build

PROGRAM = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __forceinline__ inline
static float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static float __fdividef(float a, float b) { return a / b; }
namespace c3d { constexpr float kU32 = 5.9604645e-08f; }
#include "c3d_cover.cuh"
using namespace c3d;

int main() {
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> u(0., 1.);
  long listed = 0, wrong = 0;
  for (long q = 0; q < 4000000; q++) {
    float e = (float)pow(10., -7. + 3.99 * u(g));
    unsigned b;
    memcpy(&b, &e, 4); /* bounds are bfloat16s rounded up */
    b = (b + 0xFFFFu) & 0xFFFF0000u;
    memcpy(&e, &b, 4);
    const double size = e * pow(10., 0.3 + 1.7 * u(g)), way = 6.283185307179586 * u(g), along = 3. * u(g) - 1.;
    float X[3] = {(float)(u(g) - 0.5)}, Y[3] = {(float)(u(g) - 0.5)}, err;
    X[1] = (float)(X[0] + size * cos(way));
    Y[1] = (float)(Y[0] + size * sin(way));
    const double dx = (double)X[1] - X[0], dy = (double)Y[1] - Y[0], d2 = dx * dx + dy * dy;
    double off = 0.;
    for (int k = 0; k < 5 && d2 > 0.; k++) {
      X[2] = (float)(X[0] + along * dx + off * dy);
      Y[2] = (float)(Y[0] + along * dy - off * dx);
      emit_area(X, Y, e, err);
      off = err * (1. - 3e-7 + 1.3e-6 * u(g)) / d2;
    }
    if (!(d2 > 0.) || !area_unclamped(emit_area(X, Y, e, err), err)) continue;
    listed++;
    const CoverTri c = cover_tri(X, Y, e);
    bool out, inside, far_out, far_in;
    cover_test(c, (X[0] + X[1] + X[2]) / 3.f, (Y[0] + Y[1] + Y[2]) / 3.f, out, inside);
    const float beyond = 3.f * std::max({X[0], X[1], X[2]}) - 2.f * std::min({X[0], X[1], X[2]}) + 1.f;
    cover_test(c, beyond, Y[0], far_out, far_in);
    wrong += out || far_in;
  }
  printf("%ld %ld\n", listed, wrong);
  return 0;
}
"""


def test_listed_triangles_at_the_area_bound(tmp_path):
    src, exe = tmp_path / "cover.cpp", tmp_path / "cover"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.abspath(build.CSRC), "-o", str(exe),
                    str(src)], check=True)
    listed, wrong = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert listed > 100000 and wrong == 0
