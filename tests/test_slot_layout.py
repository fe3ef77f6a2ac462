"""The shared-memory layouts (sinksim_b200/csrc/slot_layout.h, adjoint_layout.h): the largest hulls that the engine's first
layouts accepted still fit a block, in every team size that they fitted, and the places of one slot do not overlap
except where two arrays are never alive together."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sinksim_b200", "csrc")
BLOCK = 232448  # a B200 block's shared memory

SOURCE = r"""
#include "adjoint_layout.h"
#include "slot_layout.h"
#include <cstdio>
#include <cstdlib>
#include <utility>
using namespace ssb;
int main(int, char** a) {
  auto arg = [&](int k) { return std::atoi(a[k]); };
  const int nn = arg(1), nc = arg(2), ng = arg(3), mg = arg(4), W = arg(5);
  const bool mixed = arg(6), fleet = arg(7);
  const SlotLayout L = slot_layout(nn, nc, ng, mg, mixed, W, fleet);
  // (start, bytes) of every array at its largest, in the order they are placed; tmp also holds the listed connections
  const std::size_t N = 8ul * nn, lists = W <= 4 ? 2ul * nc : 0;
  const std::pair<std::uint32_t, std::size_t> at[] = {
      {L.vol, N}, {L.level, N}, {L.cx, N}, {L.cy, N}, {L.cz, N}, {L.acc, N}, {L.area, N}, {L.zmax, N}, {L.hEff, N}, {L.aEff, N},
      {L.tmp, N > lists ? N : lists}, {L.dV, 8ul * nc}, {L.passes, mg > 1 ? 40ul * mg * W * (32 / level_lanes_of(mixed, W)) : 0}, {L.hydro, 8 * 33},
      {L.misc, 4 * kMiscSlots}, {L.merged, 1ul * ng}, {L.dry, 1ul * nn}, {L.wet, (nn + 31ul) / 32}, {L.list, 2ul * ng}, {L.pose, 2 * sizeof(Pose)},
      {L.parked, sizeof(Parked)}, {fleet ? L.model : L.bytes, fleet ? sizeof(DevModel) : 0}};
  std::size_t end = 0;
  for (const auto& p : at) {
    if (p.first < end || p.first % 16) return 1;
    end = p.first + p.second;
  }
  if (end > L.bytes) return 1;
  // five columns at one stride
  const std::uint32_t stride = L.zmax - L.area;
  if (L.hEff - L.zmax != stride || L.aEff - L.hEff != stride || L.tmp - L.aEff != stride) return 1;
  const AdjLayout A = adjoint_layout(nn, nc, ng, 8, W);
  const adj::TapeLayout T = adj::tape_layout(nn, ng);
  if (A.poff < A.tape + T.doubles * 8 + T.ints * 4 || A.poff + 4ul * (nn + 1) > A.bytes || A.tape + record_bytes(T, nn, nn * adj::kMaxPasses) > A.bytes ||
      A.tape < A.sampleS + 64)
    return 1;
  const int fits = fitting_team(16, 232448, [&](int w) { return slot_layout(nn, nc, ng, mg, mixed, w, fleet); });
  std::printf("%u %zu %d\n", L.bytes, L.bytes + static_cast<std::size_t>(A.bytes), fits);
}
"""


@pytest.fixture(scope="module")
def sizes(tmp_path_factory):
    out = tmp_path_factory.mktemp("layout")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    (out / "sizes.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", include, "-I", CSRC, str(out / "sizes.cpp"), "-o", str(out / "sizes")], check=True)

    def of(*args):
        r = subprocess.run([str(out / "sizes")] + [str(int(a)) for a in args], capture_output=True, text=True)
        assert r.returncode == 0, args
        return [int(v) for v in r.stdout.split()]

    return of


# spaces, connections, spaces per group: the largest that fitted as one-warp and as 16-warp simulations
FIRST = [(2488, 0, 1, 1), (2452, 0, 1, 16), (2292, 1146, 1, 1), (2124, 2102, 1, 1), (2292, 2292, 1, 1), (2256, 2256, 1, 16), (2272, 2385, 1, 1),
         (1976, 3952, 1, 1), (1948, 3896, 1, 16), (1740, 5220, 1, 1), (1400, 7000, 1, 1), (1084, 8672, 1, 1), (2300, 2300, 2, 1), (2232, 2232, 2, 16),
         (1984, 3968, 4, 1), (1868, 3736, 4, 16), (1084, 8672, 4, 1)]


@pytest.mark.parametrize("spaces,connections,per_group,warps", FIRST)
def test_the_largest_first_hulls_fit(sizes, spaces, connections, per_group, warps):
    for mixed in (0, 1):
        assert sizes(spaces, connections, spaces // per_group, per_group, warps, mixed, 0)[0] <= BLOCK


@pytest.mark.parametrize("spaces,connections", [(2482, 0), (2286, 2286), (1972, 3944), (1398, 6990)])
def test_the_largest_first_hulls_of_a_fleet_fit(sizes, spaces, connections):
    assert sizes(spaces, connections, spaces, 1, 1, 0, 1)[0] <= BLOCK


@pytest.mark.parametrize("warps,spaces,connections", [(4, 217, 0), (8, 208, 0), (16, 191, 0), (4, 203, 203), (8, 194, 194), (16, 178, 178), (4, 189, 378),
                                                      (8, 181, 362), (16, 166, 332), (16, 118, 944)])
def test_the_largest_first_gradients_fit(sizes, warps, spaces, connections):
    assert sizes(spaces, connections, spaces, 1, warps, 0, 0)[1] <= BLOCK


@pytest.mark.parametrize("nn,nc,per_group", [(1, 0, 1), (2, 1, 2), (31, 5, 1), (32, 64, 2), (33, 400, 3), (64, 290, 2), (65, 1200, 5), (256, 700, 256)])
def test_the_places_do_not_overlap(sizes, nn, nc, per_group):
    for warps in (1, 2, 4, 8, 16):
        for mixed in (0, 1):
            for fleet in (0, 1):
                sizes(nn, nc, (nn + per_group - 1) // per_group, per_group, warps, mixed, fleet)


@pytest.mark.parametrize("group,mixed,warps", [(100, 0, 16), (184, 0, 8), (184, 1, 16), (600, 0, 2), (600, 1, 2), (1200, 0, 1)])
def test_the_largest_team_that_fits_a_large_group(sizes, group, mixed, warps):
    """A merged group's pass buffers: 40 bytes a member, lane group and team."""
    bytes_of = lambda w: sizes(group, 0, 1, group, w, mixed, 0)[0]
    assert sizes(group, 0, 1, group, 1, mixed, 0)[2] == warps
    assert bytes_of(warps) <= BLOCK and (warps == 16 or bytes_of(2 * warps) > BLOCK)
