// Which points of a set can be the lowest or the highest in the world at some attitude, bit for bit.
//
// A step needs the world extent of every flooded space (its lowest segment bottom and highest segment top) and the
// highest point of the hull. The world height of a point is computed as ((R20 x + R21 y) + tz) + R22 z, each operation
// rounded once. Rounding is monotone, so with the signs of R20 and R21 given and R22 >= 0 the computed height is
// monotone in each of x, y and z: a point can be left out when another one is no larger (for a minimum) in all three
// directed coordinates, and the minimum over the points left has the same bits as the minimum over all. The same holds
// in single precision on the rounded coordinates, because rounding a coordinate keeps the order. One list per sign
// quadrant of (R20, R21) and per end suffices; a box-shaped space keeps one corner per list (titanic64: 136 segments a
// space, 10 and 4 points on average; its 4,408 columns: 24 to 41 points).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace ssb {

// List (quadrant q, end, set n) holds points idx[start[l]] .. idx[start[l + 1]), l = (2 q + end) (sets) + n; q has bit 0
// when R20 < 0 and bit 1 when R21 < 0; end 0 the minimum of the bottoms, 1 the maximum of the tops.
struct ExtentLists {
  std::vector<std::int32_t> start, idx;
};

// A point of a set: its coordinates and index.
struct ExtentPoint {
  double x, y, z;
  std::int32_t i;
};

// Appends to out the indices of the points (in order of s z) that no other one beats in all of sx x, sy y, s z, one of
// several equal points.
inline void append_undominated(const std::vector<ExtentPoint>& from, double sx, double sy, double s, std::vector<ExtentPoint>& kept,
                               std::vector<std::int32_t>& out) {
  kept.clear();
  for (const ExtentPoint& q : from) {
    const ExtentPoint p{sx * q.x, sy * q.y, s * q.z, q.i};
    // no kept point has a larger z
    bool beaten = false;
    for (std::size_t k = kept.size(); k-- > 0 && !beaten;) beaten = kept[k].x <= p.x && kept[k].y <= p.y;
    if (beaten) continue;
    // those of the same z it beats in turn
    while (!kept.empty() && kept.back().z == p.z && p.x <= kept.back().x && p.y <= kept.back().y) kept.pop_back();
    kept.push_back(p);
  }
  for (const ExtentPoint& k : kept) out.push_back(k.i);
}

// The points of [first, first + n) without those that two neighbours in the array (one or two places away: hulls are
// stored line by line, some with the sides alternating) beat whatever the signs: the neighbours have the same x and lie on
// both sides in y, and neither is larger in s z. This leaves the ends of every flat stretch, so the lists are built from a
// fraction of the points. (Strictly on both sides, so a chain of points that beat one another ends at one that is kept.)
template <class X, class Y, class Z>
std::vector<ExtentPoint> line_ends(std::int32_t first, std::int32_t n, X x, Y y, Z z, double s) {
  std::vector<ExtentPoint> out;
  const std::int32_t end = first + n;
  auto inside = [&](std::int32_t a, std::int32_t b, std::int32_t c) {
    return a >= first && c < end && x(a) == x(b) && x(b) == x(c) && s * z(a) <= s * z(b) && s * z(c) <= s * z(b) &&
           ((y(a) < y(b) && y(b) < y(c)) || (y(a) > y(b) && y(b) > y(c)));
  };
  for (std::int32_t i = first; i < end; ++i)
    if (!inside(i - 1, i, i + 1) && !inside(i - 2, i, i + 2)) out.push_back({x(i), y(i), z(i), i});
  // the lowest (or highest) on an even keel first: a look at the first few of a list mostly settles what is asked
  std::sort(out.begin(), out.end(), [s](const ExtentPoint& a, const ExtentPoint& b) { return s * a.z < s * b.z || (a.z == b.z && a.i < b.i); });
  return out;
}

// The lists of every set n of points [start[n], start[n] + count[n]), with coordinates (x(i), y(i)), bottoms lo(i) and
// tops hi(i); sets from `tops_only` on have empty lists of bottoms.
template <class X, class Y, class Lo, class Hi>
ExtentLists extent_lists(const std::vector<std::int32_t>& start, const std::vector<std::int32_t>& count, X x, Y y, Lo lo, Hi hi,
                         std::size_t tops_only = static_cast<std::size_t>(-1)) {
  ExtentLists L;
  L.start.push_back(0);
  std::vector<std::vector<ExtentPoint>> ends[2];
  for (std::size_t n = 0; n < start.size(); ++n) {
    ends[0].push_back(line_ends(start[n], n < tops_only ? count[n] : 0, x, y, lo, 1.0));
    ends[1].push_back(line_ends(start[n], count[n], x, y, hi, -1.0));
  }
  std::vector<ExtentPoint> kept;
  for (int q = 0; q < 4; ++q)
    for (int end = 0; end < 2; ++end)
      for (std::size_t n = 0; n < start.size(); ++n) {
        // the minimum looks for small directed coordinates, the maximum for large ones
        const double s = end == 0 ? 1.0 : -1.0;
        append_undominated(ends[end][n], (q & 1) ? -s : s, (q & 2) ? -s : s, s, kept, L.idx);
        L.start.push_back(static_cast<std::int32_t>(L.idx.size()));
      }
  return L;
}

}  // namespace ssb
