// Where one simulation's state and scratch sit in its team's part of the block's shared memory.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "device_model.h"

namespace ssb {

inline std::uint32_t take(std::uint32_t& off, std::size_t bytes) {
  const std::uint32_t at = off;
  off = static_cast<std::uint32_t>((off + bytes + 15) & ~static_cast<std::size_t>(15));
  return at;
}

// The slot of one simulation of a model of these sizes, stepped by a team of W warps. Its size decides which hulls run at all
// (one slot has to fit a block's shared memory) and how much of an SM's shared storage a full load leaves to L1: 92 bytes a
// space that is a group of its own and 8 a connection, so the 232,448 bytes of a B200 block hold 2,314 spaces with as many
// connections, 2,144 with twice and 1,994 with three times as many.
// A titanic64 slot is 9.1 KB in one-warp teams. With 10.6 KB (a degree array, a sixth column of load terms and 8-byte list
// entries of their own) hulls of 1,929 to 2,292 spaces were refused that had run before, and 2,048 uneven titanic64 runs to
// 20 min took 350 ms on B200, 343 as it is; 264 liner runs to 15 min 91.7 and 89.3.
inline SlotLayout slot_layout(std::int32_t NN, std::int32_t NC, std::int32_t NG, std::int32_t maxGroup, bool mixed, int W, bool fleet) {
  SlotLayout L{};
  std::uint32_t off = 0;
  const std::size_t nb = sizeof(double) * static_cast<std::size_t>(NN);
  L.vol = take(off, nb); L.level = take(off, nb); L.cx = take(off, nb); L.cy = take(off, nb); L.cz = take(off, nb);
  L.acc = take(off, nb);
  // five columns that the loads' terms are summed down side by side, so a stride that puts them in different banks
  const std::size_t column = sizeof(double) * ((static_cast<std::size_t>(NN) + 5) / 8 * 8 + 2);
  L.area = take(off, column); L.zmax = take(off, column); L.hEff = take(off, column); L.aEff = take(off, column);
  // the last one's place also holds the list of connections (teams of up to four warps)
  L.tmp = take(off, std::max(column, W <= 4 ? sizeof(std::uint16_t) * static_cast<std::size_t>(NC) : 0));
  L.dV = take(off, sizeof(double) * static_cast<std::size_t>(std::max(NC, 1)));
  const auto levelGroups = static_cast<std::size_t>(W * (32 / level_lanes_of(mixed, W)));
  L.passes = take(off, maxGroup > 1 ? 5 * sizeof(double) * static_cast<std::size_t>(maxGroup) * levelGroups : 0);
  L.hydro = take(off, 33 * sizeof(double));
  L.misc = take(off, kMiscSlots * sizeof(std::int32_t));
  L.merged = take(off, static_cast<std::size_t>(std::max(NG, 1)));
  L.dry = take(off, static_cast<std::size_t>(std::max(NN, 1)));
  L.wet = take(off, static_cast<std::size_t>(NN) / 32 + 1);
  L.list = take(off, sizeof(std::uint16_t) * static_cast<std::size_t>(std::max(NG, 1)));
  L.pose = take(off, 2 * sizeof(Pose));
  L.parked = take(off, sizeof(Parked));
  L.model = fleet ? take(off, sizeof(DevModel)) : 0u;
  L.bytes = off;
  return L;
}

// The largest team, of up to W warps, whose slot fits `room` bytes: the pass buffers of a large group grow with the team (a
// merged group of 180 spaces fits teams of up to 8 warps). 1 when none larger does.
template <class LayoutFor>
int fitting_team(int W, std::size_t room, LayoutFor layout_for) {
  while (W > 1 && layout_for(W).bytes > room) W /= 2;
  return W;
}

}  // namespace ssb
