"""The extent lists (sinksim_b200/csrc/extents.h): the lowest bottom and highest top of a set of points over its list have
the same bits as over the whole set, at any attitude, in double and in single precision."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sinksim_b200", "csrc")

SOURCE = r"""
#include "extents.h"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace ssb;
struct P { double x, y, lo, hi; };
template <class T> T height(T r20, T r21, T r22, T tz, T x, T y, T z) { const T b = r20 * x + r21 * y + tz; return b + r22 * z; }
template <class T> bool check(const std::vector<P>& p, const std::vector<int>& start, const std::vector<int>& count, const ExtentLists& L,
                              double R20, double R21, double R22, double tz) {
  const T r20 = R20, r21 = R21, r22 = R22, t = tz;
  const int q = (R20 < 0 ? 1 : 0) + (R21 < 0 ? 2 : 0), sets = start.size();
  for (int n = 0; n < sets; ++n)
    for (int end = 0; end < 2; ++end) {
      T all = end ? -1e9 : 1e9, few = all;
      auto w = [&](int i) { return height<T>(r20, r21, r22, t, T(p[i].x), T(p[i].y), T(end ? p[i].hi : p[i].lo)); };
      for (int i = start[n]; i < start[n] + count[n]; ++i) { const T v = w(i); if (end ? v > all : v < all) all = v; }
      const int l = (2 * q + end) * sets + n;
      for (int k = L.start[l]; k < L.start[l + 1]; ++k) { const T v = w(L.idx[k]); if (end ? v > few : v < few) few = v; }
      if (!(all == few)) { std::printf("set %d end %d: %.17g against %.17g\n", n, end, double(all), double(few)); return false; }
    }
  return true;
}
int main(int, char** argv) {
  const int kind = std::atoi(argv[1]);
  std::mt19937_64 g(kind + 1);
  auto u = [&](double a, double b) { return a + (b - a) * std::uniform_real_distribution<double>(0, 1)(g); };
  std::vector<P> p;
  std::vector<int> start, count;
  for (int size : {0, 1, 2, 31, 32, 33, 136, 400}) {
    start.push_back(p.size());
    count.push_back(size);
    for (int i = 0; i < size; ++i) {
      P a;
      if (kind == 0) {         // a box on a grid, points doubled up
        a = {1.75 * ((i / 2) % 9), -8.0 + (i / 18), 3, 6};
      } else if (kind == 1) {  // a curved bottom and a sheered top on a grid
        a = {1.77 * (i % 17), 0.9 * (i / 17) - 7, 0, 0};
        a.lo = 0.01 * a.x * a.x + 0.02 * a.y * a.y; a.hi = 9 + 0.003 * a.x * a.x;
      } else {                 // a cloud
        a = {u(-140, 140), u(-14, 14), u(0, 9), u(9, 18)};
      }
      p.push_back(a);
    }
  }
  const ExtentLists L = extent_lists(start, count, [&](int i) { return p[i].x; }, [&](int i) { return p[i].y; }, [&](int i) { return p[i].lo; },
                                     [&](int i) { return p[i].hi; });
  for (int k = 0; k < 4000; ++k) {
    double th = u(-1.35, 1.35), ph = u(-1.4, 1.4);
    if (k % 4 == 1) { th *= 1e-3; ph *= 1e-3; }
    if (k % 4 == 2) { th *= 1e-17; ph *= std::pow(10.0, u(-20, 0)); }   // terms near the rounding of the others
    if (k % 8 == 3) (k % 16 == 3 ? th : ph) = 0;
    const double R20 = -std::sin(th), R21 = std::cos(th) * std::sin(ph), R22 = std::cos(th) * std::cos(ph), tz = u(-15, 2);
    if (!check<double>(p, start, count, L, R20, R21, R22, tz) || !check<float>(p, start, count, L, R20, R21, R22, tz)) return 1;
  }
  std::size_t most = 0;
  for (std::size_t l = 0; l + 1 < L.start.size(); ++l) most = std::max<std::size_t>(most, L.start[l + 1] - L.start[l]);
  std::printf("longest list %zu\n", most);
  return kind == 0 && most > 2;  // a box whose last row is cut short has two corners that can be extreme at most
}
"""


@pytest.mark.parametrize("kind", [0, 1, 2], ids=["box", "curved", "cloud"])
def test_lists_have_the_extremes_of_the_whole_sets(tmp_path, kind):
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(kind)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
