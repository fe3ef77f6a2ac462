// The batch kernel: a persistent grid whose teams (W warps each) run one simulation at a time. A team takes the
// next instance index from a device work queue (one atomicAdd), loads that instance into its shared-memory slot and
// registers, steps it until it founders, reaches tMax, meets the optional retire rule or uses up the launch's step
// budget, stores it back and takes the next one. Instances of uneven run length thus retire and admit new ones
// without a host round trip; the reference instead launched one 256-thread block per instance in fixed-size chunks
// (engine/cuda/device_step.cuh:323-434, engine/cuda/batch.cu:287-302).
//
// Adaptive team size: a launch of single-warp teams gives the most simulations per SM, but a lone simulation then
// steps slowly. When at most `yieldBelow` instances remain unfinished, the teams pause their instances and stop
// claiming; the next launch resumes them with larger teams, whose steps are several times shorter.
//
// Teams never wait on each other: the only inter-team operations are the queue's atomicAdd and the count of
// unfinished instances (atomicSub when one stops, a plain load every 64 steps).
#pragma once

#include <cuda_runtime.h>

#include "batch_kernel.h"
#include "warp_step.cuh"

namespace ssb {

constexpr int kYieldCheckEvery = 64;
// try_wait rounds a block waits for its column table to arrive before it reads the table from global memory instead
constexpr int kStageWaitLimit = 1 << 20;

// Copies the column table (xy, lh, area: ncol entries each) into the block's shared memory at dst, laid out as
// staged_columns<T>: thread 0 starts one bulk asynchronous copy per array (the part that is a whole number of 16-byte
// units; the rest, under 16 bytes, by plain copies) completing on an mbarrier after the table, and every thread waits
// for the barrier's phase with a bounded number of try_wait rounds. Returns dst, or null when the wait ran out (the
// health bit kHealthStageTimeout is set and the block reads the table from global memory). Every thread of the block
// calls it once, before the teams diverge. The sources are 256-byte aligned (TablePack).
template <class T>
__device__ const unsigned char* stage_column_table(const typename Vec2<T>::type* xy, const typename Vec2<T>::type* lh, const T* area, int ncol,
                                                   unsigned char* dst, std::int32_t* error) {
  using V2 = typename Vec2<T>::type;
  const StagedColumns<T> c = staged_columns<T>(ncol);
  const auto bar = static_cast<unsigned>(__cvta_generic_to_shared(dst + c.bytes));
  const std::size_t n = static_cast<std::size_t>(ncol);
  const std::size_t size[3] = {n * sizeof(V2), n * sizeof(V2), n * sizeof(T)};
  const unsigned char* src[3] = {reinterpret_cast<const unsigned char*>(xy), reinterpret_cast<const unsigned char*>(lh),
                                 reinterpret_cast<const unsigned char*>(area)};
  const std::size_t off[3] = {c.xy, c.lh, c.area};
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned total = 0;
    for (int k = 0; k < 3; ++k) total += static_cast<unsigned>(size[k] & ~static_cast<std::size_t>(15));
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(total) : "memory");
    for (int k = 0; k < 3; ++k) {
      const auto bulk = static_cast<unsigned>(size[k] & ~static_cast<std::size_t>(15));
      const auto to = static_cast<unsigned>(__cvta_generic_to_shared(dst + off[k]));
      if (bulk)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to), "l"(src[k]),
                     "r"(bulk), "r"(bar)
                     : "memory");
#pragma unroll 1
      for (std::size_t b = bulk; b < size[k]; ++b) dst[off[k] + b] = src[k][b];
    }
  }
  bool done = false;
#pragma unroll 1
  for (int it = 0; it < kStageWaitLimit && !done; ++it) {
    unsigned ready;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ready)
        : "r"(bar)
        : "memory");
    done = ready != 0;
  }
  if (!__syncthreads_and(done ? 1 : 0)) {
    if (threadIdx.x == 0) atomicOr(error, kHealthStageTimeout);
    return nullptr;
  }
  return dst;
}

// A trace record: the run's values by the leader, the nodes by the team's lane groups (an empty node's level is formed by
// a group's lanes side by side).
template <bool MIXED, int W>
__device__ __forceinline__ void write_record(double* rec, const SimRegs& R, const DevModel& M, const Slot& S, const Team<W>& T) {
  const int nn = M.nn;
  if (T.leader()) {
    rec[0] = R.t; rec[1] = R.zO; rec[2] = R.pitch; rec[3] = R.roll; rec[4] = R.vz; rec[5] = R.wth; rec[6] = R.wph;
    rec[7] = R.inflow; rec[8] = R.Vb; rec[9] = R.hullTop;
  }
  constexpr int LANES = kLevelLanes<MIXED, W>, GROUPS = 32 / LANES * W;
  const LevelLanes L = level_lanes<MIXED, W>(T.lane);
  double* p = rec + 10;
#pragma unroll 1
  for (int n = T.rank / LANES; n < nn; n += GROUPS) {
    const double level = group_level<MIXED, W>(M, S, n, L);
    if (L.sub == 0) {
      p[n] = S.vol[n];
      p[nn + n] = level;
      p[2 * nn + n] = S.cx[n];
      p[3 * nn + n] = S.cy[n];
      p[4 * nn + n] = S.cz[n];
    }
  }
}

// Runs one instance; returns true when the team paused it (yield) and must stop claiming.
template <bool MIXED, int W, bool FLEET>
__device__ bool run_instance(const DevModel& M, const DevBatch& B, Slot& S, int inst, const Team<W>& T) {
  constexpr int kStride = 32 * W;
  if (B.stop[inst] != kRunning) return false;
  const int rank = T.rank;
  const InstPtrs<FLEET> I{M, B, inst};
  const std::size_t iN = I.perNode();
  SimRegs R;
  {
    const double* st = B.st + static_cast<std::size_t>(inst) * 8;
    R.t = st[0]; R.zO = st[1]; R.pitch = st[2]; R.roll = st[3]; R.vz = st[4]; R.wth = st[5]; R.wph = st[6]; R.calm = st[7];
    const double* o = B.out + static_cast<std::size_t>(inst) * 7;
    R.inflow = o[0]; R.Vb = o[1]; R.hullTop = o[2]; R.mw = o[3]; R.bx = o[4]; R.by = o[5]; R.bz = o[6];
    R.foundered = B.foundered[inst];
    R.founderT = B.founderT[inst];
    R.evCount = B.evCount[inst];
  }
#pragma unroll 1
  for (int n = rank; n < M.nn; n += kStride) {
    S.vol[n] = B.vol[iN + n]; S.level[n] = B.level[iN + n];
    S.cx[n] = B.cx[iN + n]; S.cy[n] = B.cy[iN + n]; S.cz[n] = B.cz[iN + n];
    S.area[n] = 0; S.zmax[n] = 0; S.hEff[n] = 0; S.aEff[n] = 0; S.acc[n] = 0;
    S.dry[n] = 0;
  }
#pragma unroll 1
  for (int g = rank; g < M.ng; g += kStride) S.merged[g] = 0;
#pragma unroll 1
  for (int c = rank; c < M.nc; c += kStride) S.dV[c] = 0;
  T.sync();
  if (T.warp == W - 1) list_groups<true>(M, S, T.lane);
  T.sync();

  long long done = B.steps[inst];
  const long long done0 = done;
  const bool traced = inst < B.traced;
  int denseCount = 0, sampleCount = 0, curveCount = 0;
  double nextSample = 0, nextCurve = 0;
  double* denseBase = nullptr;
  double* sampleBase = nullptr;
  if (traced) {
    denseBase = B.denseRec + static_cast<std::size_t>(inst) * (B.denseSteps + 1) * B.recSize;
    sampleBase = B.sampleRec + static_cast<std::size_t>(inst) * B.maxSamples * B.recSize;
    denseCount = B.denseCount[inst]; sampleCount = B.sampleCount[inst]; nextSample = B.nextSample[inst];
  }
  if (B.curveEvery > 0) { curveCount = B.curveCount[inst]; nextCurve = B.nextCurve[inst]; }

  if (traced && done == 0 && denseCount == 0) {
    // the initial record: buoyancy at the initial pose and no inflow (the reference's Simulation::record_trace)
    const Pose F0 = make_pose(M, R.zO, R.pitch, R.roll);
    const Buoy hb = buoyancy<MIXED, W>(M, F0, T, S.hydro, S.cols);
    R.inflow = 0; R.Vb = hb.V; R.hullTop = hb.top; R.bx = hb.x; R.by = hb.y; R.bz = hb.z;
#pragma unroll 1
    for (int k = 0; k < 2; ++k) write_record<MIXED>(k == 0 ? denseBase : sampleBase, R, M, S, T);
    denseCount = 1; sampleCount = 1; nextSample = B.sampleEvery;
    T.sync();
  }

  int stop = kRunning;
  bool paused = false;
  // every thread of the team stores the same pose and values; a step replaces them (team_step)
  *S.pose = make_pose(M, R.zO, R.pitch, R.roll);
  park(S.parked, R);
  T.sync();
#pragma unroll 1
  for (long long s = 0; s < B.maxSteps; ++s) {
    if (R.foundered || R.t >= B.tMax) break;
    if (B.yieldBelow > 0 && s > 0 && (s % kYieldCheckEvery) == 0) {
      if (T.leader()) S.misc[kMiscYield] = *reinterpret_cast<volatile int*>(B.remaining) <= B.yieldBelow ? 1 : 0;
      T.sync();
      const bool y = S.misc[kMiscYield] != 0;
      T.sync();
      if (y) { paused = true; break; }
    }
    if (B.curveEvery > 0 && R.t >= nextCurve && curveCount < B.curveMax) {
      if (T.warp == 0) {
        double r7[7];
        readouts(M, R, S, r7);
        if (T.lane == 0) {
          double* rec = B.curveRec + (static_cast<std::size_t>(inst) * B.curveMax + curveCount) * 7;
          for (int k = 0; k < 7; ++k) rec[k] = r7[k];
        }
      }
      ++curveCount;
      nextCurve += B.curveEvery;
      T.sync();  // no warp starts the next solve, which changes volumes, while the first still adds them up
    }
    team_step<MIXED, W>(M, R, S, I, T);
    ++done;
    const Pose& F = *S.pose;
    if (traced) {
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        double* rec = nullptr;
        if (k == 0) {
          if (done <= B.denseSteps) rec = denseBase + static_cast<std::size_t>(denseCount++) * B.recSize;
        } else if (R.t >= nextSample - 1e-9 && sampleCount < B.maxSamples) {
          rec = sampleBase + static_cast<std::size_t>(sampleCount++) * B.recSize;
          nextSample += B.sampleEvery;
        }
        if (rec) write_record<MIXED>(rec, R, M, S, T);
      }
      T.sync();  // no warp starts the next solve while another still reads the nodes
    }
    if (B.stopWhenStable && R.t > 1800) {
      R.calm = (fabs(R.inflow) < 0.02 && fabs(R.wth) < 1e-5 && fabs(R.vz) < 1e-3) ? R.calm + M.dt : 0;
      if (R.calm > 1200) { stop = kStable; break; }
    }
    if (B.rule.enabled) {
      const double zp = world_z(F, B.rule.xDeck, B.rule.yDeck, B.rule.zDeck);
      const double zs = world_z(F, B.rule.xDeck, -B.rule.yDeck, B.rule.zDeck);
      if (fabs(R.pitch) > B.rule.pitchLimit && (zp < 0 || zs < 0)) { stop = kSinkRule; break; }
      R.calm = fabs(R.wth) < B.rule.wthLimit ? R.calm + M.dt : 0;
      if (R.calm >= B.rule.settleTime) { stop = kSettleRule; break; }
    }
  }
  if (stop == kRunning && !paused) {
    if (R.foundered) stop = kFoundered;
    else if (R.t >= B.tMax) stop = kTimeLimit;
  }

  // store the instance
  T.sync();
#pragma unroll 1
  for (int n = rank; n < M.nn; n += kStride) {
    B.vol[iN + n] = S.vol[n]; B.level[iN + n] = stale_level<MIXED>(M, S, n);
    B.cx[iN + n] = S.cx[n]; B.cy[iN + n] = S.cy[n]; B.cz[iN + n] = S.cz[n];
  }
  if (T.warp == kEventWarp<W> && T.lane == 0) B.evCount[inst] = R.evCount;
  if (T.leader()) {
    double* st = B.st + static_cast<std::size_t>(inst) * 8;
    st[0] = R.t; st[1] = R.zO; st[2] = R.pitch; st[3] = R.roll; st[4] = R.vz; st[5] = R.wth; st[6] = R.wph; st[7] = R.calm;
    double* o = B.out + static_cast<std::size_t>(inst) * 7;
    o[0] = R.inflow; o[1] = R.Vb; o[2] = R.hullTop; o[3] = R.mw; o[4] = R.bx; o[5] = R.by; o[6] = R.bz;
    B.foundered[inst] = R.foundered;
    B.founderT[inst] = R.founderT;
    B.steps[inst] = done;
    B.stop[inst] = stop;
    if (!(isfinite(R.zO) && isfinite(R.pitch) && isfinite(R.roll) && isfinite(R.vz) && isfinite(R.wth) && isfinite(R.wph)))
      atomicOr(B.error, kHealthNonFinite);
    if (traced) { B.denseCount[inst] = denseCount; B.sampleCount[inst] = sampleCount; B.nextSample[inst] = nextSample; }
    if (B.curveEvery > 0) { B.curveCount[inst] = curveCount; B.nextCurve[inst] = nextCurve; }
    if (stop != kRunning) atomicSub(B.remaining, 1);
    if (B.phaseSteps) atomicAdd(B.phaseSteps, static_cast<unsigned long long>(done - done0));
  }
  if (stop != kRunning && T.warp == 0) {
    double r7[7];
    readouts(M, R, S, r7);
    if (T.lane == 0)
      for (int k = 0; k < 7; ++k) B.finalRec[static_cast<std::size_t>(inst) * 7 + k] = r7[k];
  }
  T.sync();
  return paused;
}

// The persistent batch kernel: teams claim instances from the work queue until it runs dry (or the phase yields). In a
// fleet (FLEET), a team first copies its instance's model description into its slot and steps the instance with it.
template <bool MIXED, int W, bool FLEET>
__global__ void __launch_bounds__(kMaxWarpsPerBlock * 32, kMinBlocksPerSM) run_batch(const __grid_constant__ DevModel M, const __grid_constant__ DevBatch B, const __grid_constant__ SlotLayout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warpInBlock = threadIdx.x >> 5;
  const int team = warpInBlock / W;
  Team<W> T;
  T.warp = warpInBlock % W;
  T.lane = threadIdx.x & 31;
  T.rank = T.warp * 32 + T.lane;
  T.bar = team + 1;
  unsigned char* const slot = smem + static_cast<std::size_t>(team) * L.bytes;
  Slot S = carve_slot(slot, L);
  if constexpr (!FLEET) {
    if (B.stageColumns) {
      // the column table after the block's slots (one copy per block for the whole launch)
      unsigned char* const table = smem + static_cast<std::size_t>(blockDim.x / (32 * W)) * L.bytes;
      if constexpr (MIXED) S.cols = stage_column_table<float>(M.colXYf, M.colLHf, M.colAf, M.ncol, table, B.error);
      else S.cols = stage_column_table<double>(M.colXY, M.colLH, M.colA, M.ncol, table, B.error);
    }
  }
  for (;;) {
    if (T.leader()) {
      const int q = atomicAdd(B.queue, 1);
      S.misc[kMiscInstance] = B.order == nullptr ? q : (q < *B.orderCount ? B.order[q] : B.count);
      S.misc[kMiscTaken] = W * (32 / kLevelLanes<MIXED, W>);  // the level solve's list counter for the first step (team_step resets it)
    }
    T.sync();
    const int inst = S.misc[kMiscInstance];
    T.sync();
    if (inst >= B.count) return;
    if constexpr (FLEET) {
      static_assert(sizeof(DevModel) % sizeof(unsigned) == 0, "the model description is copied in 32-bit words");
      DevModel* const own = reinterpret_cast<DevModel*>(slot + L.model);
      const unsigned* src = reinterpret_cast<const unsigned*>(B.models + B.model[inst]);
      unsigned* dst = reinterpret_cast<unsigned*>(own);
#pragma unroll 1
      for (int k = T.rank; k < static_cast<int>(sizeof(DevModel) / sizeof(unsigned)); k += 32 * W) dst[k] = src[k];
      T.sync();
      // run_instance ends with a team barrier, so no thread still reads this copy when the next claim overwrites it
      if (run_instance<MIXED, W, true>(*own, B, S, inst, T)) return;
    } else {
      if (run_instance<MIXED, W, false>(M, B, S, inst, T)) return;
    }
  }
}

// The host side of one instantiation of the kernel. Each is compiled in a unit of its own (batch_kernel_inst.cu), so that
// a build spreads them over its processes; batch_kernel.cu dispatches to them.
template <bool MIXED, int W, bool FLEET>
struct BatchKernel {
  static cudaError_t set_smem(std::size_t bytes);
  static cudaError_t occupancy(int threads, std::size_t bytes, int* perSM);
  static void launch(const DevModel& M, const DevBatch& B, const SlotLayout& L, int grid, int threads, std::size_t smem, cudaStream_t s);
};

}  // namespace ssb
