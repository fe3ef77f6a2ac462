// Device-side layout of one compiled model (ship + sim) and of a batch of its instances.
//
// Layout in HBM. Everything a step reads from the model is structure-of-arrays so that a warp reading entries
// j..j+31 moves whole 128-byte lines:
//   columns   x, y, dxdy, zlo, zhi                     [ncol] f64       the buoyancy clip (hydro pass)
//   segments  x, y, A (= dxdy of the column), a, e     [nseg] f64       the node pass, with the column gather of the
//                                                                       reference (segCol -> x, y, dxdy) resolved once
//                                                                       on the host, so a segment visit has no
//                                                                       dependent load
//   nodes, groups, connections, incidence (CSR), monitor lists (CSR), marks: small tables read through L1.
// Per instance (count instances): the connection fields a sweep may change (en, area, tOn), the state (t, pose,
// rates, per-node volume, level and centroid), the outputs, the event log, the readout curve and, for the first
// `traced` instances, the trace records. The state of an instance being stepped lives in shared memory and
// registers of its warp; global memory holds it between launches and after the run.
#pragma once

#include <cstdint>

#include <vector_types.h>

namespace ssb {

// A group as a step's level solve takes it, in one load: its first two members (a group of one: that one twice), their number
// (255: at least that many) and its merge mode.
struct alignas(8) GroupEntry {
  std::uint16_t n0, n1;
  std::uint8_t N, mode;
};

struct DevModel {
  // columns: (x, y) and (zlo, zhi) pairs, so one 16-byte load fetches two fields, and the footprint dxdy; the float
  // copies are the same values rounded to single precision once on the host (the portable32 column arithmetic
  // rounds every geometry value to float before using it, kernel/reduce.hpp:131-164)
  std::int32_t ncol;
  const double2 *colXY, *colLH;
  const double* colA;
  const float2 *colXYf, *colLHf;
  const float* colAf;
  // segments with the column gather resolved: (x, y) of the column, (a, e) of the segment, the column's dxdy
  std::int32_t nseg;
  const double2 *segXY, *segLH;
  const double* segAr;
  const float2 *segXYf, *segLHf;
  const float* segArf;
  // extent lists (extents.h) of the nodes' segments and, as set nn, of the hull columns' tops: 8 (nn + 1) + 1 starts and
  // the listed points' coordinates, (x, y) and z
  const std::int32_t* exStart;
  const double2* exXY;
  const double* exZ;
  const float2* exXYf;
  const float* exZf;
  // nodes
  std::int32_t nn;
  const double *mu, *vmax, *amin, *aov;
  const std::int32_t *segStart, *segCount;
  const int2* nodeSeg;  // (segStart, segCount)
  // groups
  std::int32_t ng;
  const std::int32_t *gStart, *gCount, *gNodes;
  const GroupEntry* groupEntry;
  const double *gpx, *gpy, *gpz;
  double gMargin;
  std::int32_t maxGroup;
  // connections (the immutable fields)
  std::int32_t nc;
  const std::int32_t *ca, *cb, *skip;
  const std::uint8_t* law;
  const double *kx, *ky, *kz, *coef;
  // incidence: per node its connections in increasing order (side 1 at the b end), and the sea connections
  const std::int32_t *incStart, *incCount, *incConn;
  const std::uint8_t* incSide;
  const std::int32_t* incEdge;  // 2 incConn + incSide
  std::int32_t nsea;
  const std::int32_t* sea;
  // monitors: per monitor its connections in increasing order
  std::int32_t nmon;
  double monThreshold;
  const std::int32_t *monStart, *monCount, *monConn;
  // marks
  std::int32_t nmark;
  const double *mkx, *mky, *mkz;
  const std::uint8_t* mkWhen;
  // founder rule
  double hullTopBelow, pitchAbsAbove, buoyancyBelow, minT;
  // physics and body
  double rho, g, sq2g, dt;
  double ms, g0x, g0y, g0z, XO, YO, mh0, Ith0, Iph0, cDz, cDth, cDph, qz, qth, qph;
  // readout geometry
  double xFP, xAP;
  std::int32_t evCap;
};

// An extra retire predicate evaluated after every step (the batching workloads' "sink" and "settle" rules); it
// never changes the physics. Disabled when enabled == 0.
struct RetireRule {
  std::int32_t enabled;
  double pitchLimit;           // rad: sink when |pitch| exceeds this ...
  double xDeck, yDeck, zDeck;  // ... and the deck edge at (xDeck, +-yDeck, zDeck) is below the sea
  double wthLimit;             // rad/s: settle when |pitch rate| stays below this ...
  double settleTime;           // s: ... for this long
};

// Why an instance stopped. kStable: the reference's "stop when stable" calm rule of Simulation::run
// (engine/src/simulation.cpp:179-182), which its GPU runner refused (apps/sinksim_cuda_run.cpp:28).
enum StopReason : std::int32_t { kRunning = 0, kFoundered = 1, kTimeLimit = 2, kSinkRule = 3, kSettleRule = 4, kStable = 5 };

// Bits of DevBatch::error, which a batch run reports to the host: kHealthNonFinite, an instance's rigid-body state
// (heave, pitch, roll or their rates) was not finite when the kernel stored it (a NaN or infinity in an input, or a
// model that diverged). The physics is not changed by it: the instance's results are what the step computed.
// kHealthStageTimeout: a block's copy of the column table into shared memory (stageColumns) did not complete within
// its wait limit; that block read the table from global memory instead, with the same results.
enum HealthBit : std::int32_t { kHealthNonFinite = 1, kHealthStageTimeout = 2 };

struct DevBatch {
  std::int32_t count;
  // connection fields per instance [count * nc]
  const std::uint8_t* en;
  const double* area;
  const double* tOn;
  // state per instance
  double* st;       // [count * 8]: t, zO, pitch, roll, vz, wth, wph, calm (seconds the settle rule has held)
  double* out;      // [count * 7]: inflow, Vb, hullTop, mw, bx, by, bz
  double *vol, *level, *cx, *cy, *cz;   // [count * nn]
  // events
  double* evT;             // [count * evCap]
  std::int32_t* evId;      // [count * evCap]
  std::int32_t* evKind;    // [count * evCap]
  std::int32_t* evCount;   // [count]
  double* overT;           // [count * nmon]
  double* markT;           // [count * nmark]
  std::int32_t* foundered; // [count]
  double* founderT;        // [count]
  long long* steps;        // [count]
  std::int32_t* stop;      // [count] StopReason
  // readout curve of every instance: 7 values per record when t >= nextCurve
  double curveEvery;       // <= 0 disables
  std::int32_t curveMax;
  double* curveRec;        // [count * curveMax * 7]
  std::int32_t* curveCount;
  double* nextCurve;
  // final readouts of every instance, computed on the device when the instance stops: 7 values
  double* finalRec;        // [count * 7]
  // traces of the first `traced` instances
  std::int32_t traced, denseSteps, maxSamples, recSize;
  double sampleEvery;
  double *denseRec, *sampleRec;
  std::int32_t *denseCount, *sampleCount;
  double* nextSample;
  // run control
  double tMax;
  long long maxSteps;          // steps per instance per launch
  std::int32_t firstLaunch;
  RetireRule rule;
  // the reference's calm rule: after 1,800 s, stop once |inflow| < 0.02, |pitch rate| < 1e-5 and |heave rate| < 1e-3
  // have held for more than 1,200 s; exclusive with `rule` (both keep their timer in state slot 7)
  std::int32_t stopWhenStable;
  std::int32_t* queue;         // work-queue head (atomic), reset to 0 before each launch
  std::int32_t* error;         // HealthBit flags of the run (0 = none), or-ed by the kernels and read back by the host
  // 1: every block first copies the model's column table (the arrays the buoyancy reads, in the arithmetic's type)
  // into its shared memory after its slots, by bulk asynchronous copies, and the buoyancy reads it from there
  std::int32_t stageColumns;
  // adaptive team size: instances not yet stopped (atomic, set to count before the first launch); a launch with
  // yieldBelow > 0 pauses its instances and stops claiming new ones once at most yieldBelow remain, so that the
  // next launch resumes them with larger teams (shorter steps)
  std::int32_t* remaining;
  std::int32_t yieldBelow;
  // when not null: the steps this launch took, summed over its instances (the per-phase work figure of the timing)
  unsigned long long* phaseSteps;
  // when not null: queue position k claims instance order[k] (k < *orderCount) instead of instance k. Launch phases
  // after the first take the unfinished instances with the fewest steps done first, so that the runs with the most
  // work left to do are the first to get the larger teams.
  const std::int32_t* order;
  const std::int32_t* orderCount;
  // A fleet (instances of several models in one launch): instance i steps models[model[i]], and its per-node,
  // per-connection, event, monitor and mark arrays start at the offsets below instead of i x the model's size.
  // Null for a batch of one model, which the kernel's model parameter describes.
  const DevModel* models;
  const std::int32_t* model;
  const long long *nodeOff, *connOff, *evOff, *monOff, *markOff;
};

// Pose R = Ry(pitch) Rx(roll) and translation (kernel/frame.hpp:9-21), with the single-precision copies the
// portable32 column arithmetic uses (kernel/reduce.hpp:86-98). A team keeps the pose of its current step in its slot.
struct Pose {
  double R00, R01, R02, R10, R11, R12, R20, R21, R22, tx, ty, tz, cth, iR;
  float fR20, fR21, fR22, ftz, fiR;
};

// The buoyancy pass's result: displaced volume, its centroid in the ship frame, the highest hull point in the world.
struct Buoy {
  double V, x, y, z, top;
};

// The run's values, which a team keeps in its slot through a step, so that their registers serve its phases.
struct Parked {
  double t, zO, pitch, roll, vz, wth, wph, inflow, Vb, hullTop, mw, bx, by, bz, founderT;
  int foundered;
};

// Lanes that solve one group of nodes' free-surface levels together (16 or 32), per numerics and team size: a warp works
// on 32 / kLevelLanes groups at once. Each lane forms the partials of 32 / kLevelLanes lanes of the 32-lane node-pass tree
// and combines them in the tree's order, so the results do not depend on this choice. Fewer lanes per group give more
// groups in flight and fewer shuffles, more lanes a shorter chain per pass. On B200 (16 lanes against the other choice):
// double precision, 8-warp teams, 264 liner runs to 15 min 95.0 ms, 88.6 with 32; 16-warp teams, 192 titanic64 runs to
// 1 h 266, 273 with 32; 1- and 2-warp teams, 2,048 uneven runs 348, 371 with 32, 359 with 8. Single precision, small
// teams, 1,021 uneven runs 143, 161 with 8, 145 with 32; large teams, 48 runs 49.7, 45.7 with 32.
constexpr int level_lanes_of(bool mixed, int W) { return mixed ? (W >= 8 ? 32 : 16) : (W == 8 ? 32 : 16); }
template <bool MIXED, int W>
constexpr int kLevelLanes = level_lanes_of(MIXED, W);

// A slot's small team values: the claimed instance, the yield flag, the level solve's counter of list entries taken, the
// list's length, the numbers of flows at the front and at the back of their list.
enum MiscSlot { kMiscInstance = 0, kMiscYield = 1, kMiscTaken = 2, kMiscListed = 3, kMiscFront = 4, kMiscBack = 5, kMiscSlots = 6 };

// Byte offsets of one simulation slot (one team of warps) in dynamic shared memory; `bytes` is the slot stride
// (slot_layout.h lays it out). passes holds maxGroup node-pass results per level lane group of the team, in models that have
// groups of more than one; hydro the eight buoyancy tree results and the hull's top; misc the team's small broadcast values
// and counters (MiscSlot); dry a flag byte per node, wet the numbers of load terms, list the groups the next level solve
// visits (warp_step.cuh); pose this step's pose and the last one's, which every phase reads (kept here rather than in each
// thread's registers); parked the run's values; model (fleets only) the team's copy of its instance's model. Arrays serve
// more than one phase of a step: between the level solve and the heads acc, hEff, aEff and tmp hold the passes' sums; then,
// until the volume update, acc holds the nodes' degrees and tmp's place the list of the connections that can flow; then acc
// holds the excess, and area, zmax, hEff, aEff and tmp are the five columns of the loads' terms (a fixed stride apart).
struct SlotLayout {
  std::uint32_t vol, level, cx, cy, cz, area, zmax, hEff, aEff, tmp, acc, dV, passes, hydro, misc, merged, dry, wet, list, pose, parked, model, bytes;
};

}  // namespace ssb
