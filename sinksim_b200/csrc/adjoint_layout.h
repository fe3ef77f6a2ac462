// Sizes of the adjoint's packed step records, and where a team's reverse arrays sit in shared memory after its forward slot.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "adjoint_kernel.h"
#include "adjoint_step.cuh"

namespace ssb {

// A packed step record: the tape's int32 (pass counts, merged flags), each node's first pass record in the packed
// order and their total (nn + 1 int32; padded to 8 bytes), the tape's doubles up to the pass records, then only the
// pass records the step used, node by node (min(count, kMaxPasses) per node), the whole rounded up to 16 bytes. The
// pass records dominate the unpacked tape (kMaxPasses slots per node), and a node takes about 1.2 passes per step, so a
// record is about a third of the tape; the stored offsets let its reader place every pass without a scan.
SSB_HD std::size_t record_ints_bytes(const adj::TapeLayout& L, int nn) {
  return ((L.ints + static_cast<std::size_t>(nn) + 1) * sizeof(std::int32_t) + 7) & ~static_cast<std::size_t>(7);
}

SSB_HD std::size_t record_bytes(const adj::TapeLayout& L, int nn, int records) {
  return (record_ints_bytes(L, nn) + (L.passes + static_cast<std::size_t>(records) * adj::kPassFields) * sizeof(double) + 15) &
         ~static_cast<std::size_t>(15);
}

// withRaw: room for one packed step record of the largest size (the reverse's asynchronous copy of the next record)
inline AdjLayout adjoint_layout(int nn, int nc, int ng, int nsamples, int W, bool withRaw = false) {
  AdjLayout A{};
  std::uint32_t off = 0;
  auto take16 = [&](std::size_t bytes) {
    const std::uint32_t at = off;
    off = static_cast<std::uint32_t>((off + bytes + 15) & ~static_cast<std::size_t>(15));
    return at;
  };
  const std::size_t N = sizeof(double) * static_cast<std::size_t>(std::max(nn, 1));
  const std::size_t C = sizeof(double) * static_cast<std::size_t>(std::max(nc, 1));
  A.hEff = take16(N); A.aEff = take16(N); A.dV = take16(C); A.volPost = take16(N);
  A.deg = take16(sizeof(int) * static_cast<std::size_t>(std::max(nn, 1)));
  A.clip = take16(sizeof(std::int32_t) * static_cast<std::size_t>(std::max(nn, 1)));
  A.aVolPost = take16(N); A.aCxs = take16(N); A.aCys = take16(N); A.aCzs = take16(N); A.aVs = take16(N); A.aAcc = take16(N);
  A.aZmx = take16(N); A.aLs = take16(N); A.aAs = take16(N);
  A.faHA = take16(C); A.faHB = take16(C); A.faAA = take16(C); A.faAB = take16(C);
  A.red = take16(sizeof(double) * 16 * static_cast<std::size_t>(W));
  A.work = take16(sizeof(adj::UnitWork) * static_cast<std::size_t>(W));
  A.plain = take16(static_cast<std::size_t>(std::max(nn, 1)));
  A.units = take16(sizeof(std::int32_t) * static_cast<std::size_t>(std::max(nn, 1)));
  A.nunits = take16(sizeof(std::int32_t));
  A.pw = take16(2 * C);
  A.replays = take16(sizeof(adj::Replay) * static_cast<std::size_t>(std::max(nn, 1)));
  A.raw = withRaw ? take16(record_bytes(adj::tape_layout(nn, ng), nn, nn * adj::kMaxPasses)) : 0;
  A.aVol = take16(N); A.aLevel = take16(N); A.aCx = take16(N); A.aCy = take16(N); A.aCz = take16(N);
  A.grad = take16(C);
  A.sampleS = take16(sizeof(double) * static_cast<std::size_t>(std::max(nsamples, 1)));
  // a step's tape with the packing offsets behind it; at another time, over both, a packed record of the largest size
  const adj::TapeLayout TL = adj::tape_layout(nn, ng);
  const std::size_t offsets = sizeof(std::int32_t) * (static_cast<std::size_t>(std::max(nn, 1)) + 1);
  A.tape = take16(std::max(TL.bytes + offsets, record_bytes(TL, nn, nn * adj::kMaxPasses)));
  A.poff = A.tape + static_cast<std::uint32_t>(TL.bytes);
  A.bytes = off;
  return A;
}

}  // namespace ssb
