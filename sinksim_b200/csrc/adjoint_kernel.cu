// The adjoint kernel: the gradient of a trajectory objective with respect to every connection area, for a batch of
// instances, by a hand-written discrete adjoint of the time step with checkpoints (no counterpart in the reference,
// which has no gradients: docs/adr/0001-single-source-cpp-kernel.md:25-26).
//
// A persistent grid of teams (W warps each, one instance at a time from a work queue), per instance:
//   1. forward: the instance runs from its initial state to tMax or its founder, exactly as the batch kernel steps it
//      (the same team_step, so the same bits), keeping the state every K steps (a checkpoint: t, pose, rates and every
//      node's volume, level and centroid, FP64) and the objective's readouts at the sample times. With the tape hooks
//      on (tapeForward), every step's tape (every node pass of the level solve, the solved levels, pose and buoyancy)
//      goes to shared memory and from there, packed, into the team's ring of step records in global memory;
//   2. reverse: segment by segment, last first. A segment whose records the ring still holds is reversed from them;
//      any other is recomputed from its checkpoint with the tape hooks on, into the ring, first. Each step's record is
//      copied into shared memory as it is and reversed there (adjoint_step.cuh), adding the objective's adjoint at the
//      sample states.
// Memory per team: the checkpoints of one run and the ring; the adjoint of the state lives in shared memory. When the
// ring holds a whole run (the usual case: a packed record is about 12 KB on a 64-node model) nothing is recomputed;
// with a ring of K records every segment is recomputed once, which costs one more forward pass.
//
// The objective: J = sum_k (trim(s_k) - trim*_k)^2 + (heave(s_k) - heave*_k)^2, trim in degrees and heave the mean of
// the forward and aft drafts, where s_k is the state at which a readout curve recorded every sample time would take its
// record (the first step start with t >= t_k; the final state for a run that stopped before t_k).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "adjoint_kernel.h"
#include "adjoint_layout.h"
#include "adjoint_step.cuh"
#include "warp_step.cuh"

namespace ssb {

namespace {

using adj::AdjPose;
using adj::PoseD;

template <int W>
struct AdjTeam {
  int rank, size, warp, nwarps, lane, width, bar;
  __device__ __forceinline__ void sync() const {
    if constexpr (W == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(W * 32) : "memory");
  }
  __device__ __forceinline__ void add_int(int* p, int v) const { atomicAdd(p, v); }
  // team-wide sums of K values (K <= 16), every thread receives them. The lanes' butterfly (offsets 16 .. 1) halves the
  // values a lane carries at each of its first four offsets, so 31 exchanges do for 16 values instead of 80, with the same
  // pairs at every offset and so the same bits; each warp's sums go through shared memory, lane k of every warp adds value
  // k over the warps (in warp order) and the lanes pass the K totals round.
  template <int K>
  __device__ __forceinline__ void reduce(double (&v)[K], int, double* red) const {
    static_assert(K <= 16, "at most 16 values");
    double x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = k < K ? v[k] : 0.0;
    int mine = 0;  // the value this lane ends with
#pragma unroll
    for (int off = 16, n = 16; off > 1; off >>= 1, n >>= 1) {
      const bool upper = (lane & off) != 0;
#pragma unroll
      for (int k = 0; k < n / 2; ++k) {
        const double keep = upper ? x[k + n / 2] : x[k], give = upper ? x[k] : x[k + n / 2];
        x[k] = keep + __shfl_xor_sync(0xffffffffu, give, off);
      }
      if (upper) mine += n / 2;
    }
    x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
    if (mine < K && (lane & 1) == 0) red[warp * 16 + mine] = x[0];
    sync();
    double s = 0;
    if (lane < K)
#pragma unroll 4
      for (int w = 0; w < W; ++w) s += red[w * 16 + lane];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = __shfl_sync(0xffffffffu, s, k);
    sync();
  }
};

// The tape hooks of the forward step (NoTape's counterpart): one lane of a level lane group writes each node pass, the
// team writes the solved state, the pose and the buoyancy result.
struct GpuTape {
  static constexpr bool kLazy = false;  // every level is formed: records and checkpoints keep them
  adj::Tape t;
  bool on;  // false: the step is not recorded
  // A unit's start: its first pass's level and extent; the sums stay zero when no pass is made there.
  __device__ __forceinline__ void start(int n, double h, double zmin, double zmax, const LevelLanes& L) const {
    if (!on || L.sub != 0) return;
    double* r = t.pass(n, 0);
    r[0] = h; r[1] = 0; r[2] = 0; r[3] = 0; r[4] = 0; r[5] = 0; r[6] = zmin; r[7] = zmax;
    t.i[t.L.npass + n] = 1;
  }
  __device__ __forceinline__ void pass(int n, int k, double h, const PassR& p, const LevelLanes& L) const {
    if (!on || L.sub != 0) return;
    if (k < adj::kMaxPasses) {
      const double* r0 = t.pass(n, 0);
      const double zmin = r0[6], zmax = r0[7];
      double* r = t.pass(n, k);
      r[0] = h; r[1] = p.vol; r[2] = p.dv; r[3] = p.mx; r[4] = p.my; r[5] = p.mz; r[6] = zmin; r[7] = zmax;
    }
    t.i[t.L.npass + n] = k + 1;
  }
  template <int W>
  __device__ __forceinline__ void solved(const DevModel& M, const Slot& S, const Team<W>& T) const {
    if (!on) return;
    const adj::TapeLayout& L = t.L;
    for (int n = T.rank; n < M.nn; n += 32 * W) {
      t.d[L.volS + n] = S.vol[n]; t.d[L.levelS + n] = S.level[n]; t.d[L.areaS + n] = S.area[n];
      t.d[L.cxS + n] = S.cx[n]; t.d[L.cyS + n] = S.cy[n]; t.d[L.czS + n] = S.cz[n]; t.d[L.zmaxS + n] = S.zmax[n];
    }
    for (int g = T.rank; g < M.ng; g += 32 * W) t.i[L.merged + g] = S.merged[g];
    if (T.leader()) {
      const Pose& F = *S.pose;
      const double p[14] = {F.R00, F.R01, F.R02, F.R10, F.R11, F.R12, F.R20, F.R21, F.R22, F.tx, F.ty, F.tz, F.cth, F.iR};
      for (int k = 0; k < 14; ++k) t.d[L.pose + k] = p[k];
      const Buoy b = buoyancy_finish(S.hydro);
      t.d[L.buoy] = b.V; t.d[L.buoy + 1] = b.x; t.d[L.buoy + 2] = b.y; t.d[L.buoy + 3] = b.z;
    }
  }
};

// Instance fields for team_step: the connection fields of the instance; events go nowhere (the adjoint runs keep no
// event log: the founder flag, which ends a run, is kept in registers by team_step itself).
struct AdjInst {
  const std::uint8_t* en_;
  const double *area_, *tOn_;
  double* sink;  // per team: evCap + nmon + nmark doubles that absorb the event bookkeeping
  std::int32_t* isink;
  int nmon;
  __device__ __forceinline__ const std::uint8_t* en() const { return en_; }
  __device__ __forceinline__ const double* area() const { return area_; }
  __device__ __forceinline__ const double* tOn() const { return tOn_; }
  __device__ __forceinline__ double* evT() const { return sink; }
  __device__ __forceinline__ std::int32_t* evId() const { return isink; }
  __device__ __forceinline__ std::int32_t* evKind() const { return isink; }
  __device__ __forceinline__ double* overT() const { return sink; }
  __device__ __forceinline__ double* markT() const { return sink + nmon; }
};

// Per-team shared memory: the forward slot, then the reverse's arrays.
struct AdjSmem {
  unsigned char* raw;   // another packed record (stageRecords), or null
  adj::RevSlot rs;
  adj::AdjState as;
  double* grad;      // [nc]
  double* sampleS;   // [nsamples] state index of each sample (as doubles)
  unsigned char* tape;  // one step's tape, written by the step's hooks; in the reverse a packed record
  std::int32_t* poff;   // [nn + 1] first pass record of each node in a packed record, then their total
};

__device__ __forceinline__ AdjSmem carve_adjoint(unsigned char* base, const AdjLayout& A) {
  AdjSmem m;
  auto d = [&](std::uint32_t off) { return reinterpret_cast<double*>(base + off); };
  m.rs.hEff = d(A.hEff); m.rs.aEff = d(A.aEff); m.rs.dV = d(A.dV); m.rs.volPost = d(A.volPost);
  m.rs.deg = reinterpret_cast<int*>(base + A.deg);
  m.rs.clip = reinterpret_cast<std::int32_t*>(base + A.clip);
  m.rs.aVolPost = d(A.aVolPost); m.rs.aCxs = d(A.aCxs); m.rs.aCys = d(A.aCys); m.rs.aCzs = d(A.aCzs); m.rs.aVs = d(A.aVs);
  m.rs.aAcc = d(A.aAcc); m.rs.aZmx = d(A.aZmx); m.rs.aLs = d(A.aLs); m.rs.aAs = d(A.aAs);
  m.rs.faHA = d(A.faHA); m.rs.faHB = d(A.faHB); m.rs.faAA = d(A.faAA); m.rs.faAB = d(A.faAB);
  m.rs.red = d(A.red);
  m.rs.work = reinterpret_cast<adj::UnitWork*>(base + A.work);
  m.rs.plain = base + A.plain;
  m.rs.units = reinterpret_cast<std::int32_t*>(base + A.units);
  m.rs.nunits = reinterpret_cast<std::int32_t*>(base + A.nunits);
  m.rs.pw = d(A.pw);
  m.rs.replays = reinterpret_cast<adj::Replay*>(base + A.replays);
  m.as.aVol = d(A.aVol); m.as.aLevel = d(A.aLevel); m.as.aCx = d(A.aCx); m.as.aCy = d(A.aCy); m.as.aCz = d(A.aCz);
  m.grad = d(A.grad);
  m.sampleS = d(A.sampleS);
  m.tape = base + A.tape;
  m.raw = A.raw ? base + A.raw : nullptr;
  m.poff = reinterpret_cast<std::int32_t*>(base + A.poff);
  return m;
}

// A checkpoint: t, zO, pitch, roll, vz, wth, wph, then vol, level, cx, cy, cz per node.
template <int W>
__device__ __forceinline__ void save_state(double* c, const SimRegs& R, const Slot& S, int nn, const Team<W>& T) {
  if (T.leader()) { c[0] = R.t; c[1] = R.zO; c[2] = R.pitch; c[3] = R.roll; c[4] = R.vz; c[5] = R.wth; c[6] = R.wph; }
  for (int n = T.rank; n < nn; n += 32 * W) {
    c[7 + n] = S.vol[n]; c[7 + nn + n] = S.level[n]; c[7 + 2 * nn + n] = S.cx[n]; c[7 + 3 * nn + n] = S.cy[n]; c[7 + 4 * nn + n] = S.cz[n];
  }
}

// Loads a state into the team's registers and slot, with the step's scratch cleared (as the batch kernel does when it
// claims an instance).
template <int W>
__device__ __forceinline__ void load_state(const double* c, SimRegs& R, Slot& S, const DevModel& M, const Team<W>& T) {
  R.t = c[0]; R.zO = c[1]; R.pitch = c[2]; R.roll = c[3]; R.vz = c[4]; R.wth = c[5]; R.wph = c[6];
  R.calm = 0; R.inflow = 0; R.Vb = 0; R.hullTop = 0; R.mw = 0; R.bx = 0; R.by = 0; R.bz = 0;
  R.foundered = 0; R.founderT = -1;
  R.evCount = M.evCap;  // no event is recorded
  const int nn = M.nn;
  for (int n = T.rank; n < nn; n += 32 * W) {
    S.vol[n] = c[7 + n]; S.level[n] = c[7 + nn + n]; S.cx[n] = c[7 + 2 * nn + n]; S.cy[n] = c[7 + 3 * nn + n]; S.cz[n] = c[7 + 4 * nn + n];
    S.area[n] = 0; S.zmax[n] = 0; S.hEff[n] = 0; S.aEff[n] = 0; S.acc[n] = 0;
    S.dry[n] = 0;
  }
  for (int g = T.rank; g < M.ng; g += 32 * W) S.merged[g] = 0;
  for (int c2 = T.rank; c2 < M.nc; c2 += 32 * W) S.dV[c2] = 0;
  T.sync();
  if (T.warp == W - 1) list_groups<false>(M, S, T.lane);  // every group, for the whole run
  T.sync();
}

// poff[n] = the first pass record of node n in the packed order, poff[nn] = their total (warp 0 scans the counts).
template <int W>
__device__ __forceinline__ void pass_offsets(const std::int32_t* npass, int nn, std::int32_t* poff, const Team<W>& T) {
  if (T.warp == 0) {
    int carry = 0;
    for (int base = 0; base < nn; base += 32) {
      const int n = base + T.lane;
      const int v = n < nn ? min(npass[n], adj::kMaxPasses) : 0;
      int x = v;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (T.lane >= o) x += y;
      }
      if (n < nn) poff[n] = carry + x - v;
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
    if (T.lane == 0) poff[nn] = carry;
  }
  T.sync();
}

// Packs the step's tape (shared memory) into dst (global); returns the record's bytes. Every thread of the team calls
// it; the tape may be overwritten once it returns.
template <int W>
__device__ __forceinline__ std::size_t store_record(const adj::Tape& tp, int nn, std::int32_t* poff, unsigned char* dst, const Team<W>& T) {
  const adj::TapeLayout& L = tp.L;
  pass_offsets(tp.i + L.npass, nn, poff, T);
  std::int32_t* di = reinterpret_cast<std::int32_t*>(dst);
  for (std::size_t i = T.rank; i < L.ints; i += 32 * W) di[i] = tp.i[i];
  for (int n = T.rank; n <= nn; n += 32 * W) di[L.ints + n] = poff[n];
  double* dd = reinterpret_cast<double*>(dst + record_ints_bytes(L, nn));
  for (std::size_t i = T.rank; i < L.passes; i += 32 * W) dd[i] = tp.d[i];
  // a round per pass number: nodes take one or two passes, so later rounds are empty and end the loop
  for (int k = 0;; ++k) {
    bool more = false;
    for (int i = T.rank; i < nn * adj::kPassFields; i += 32 * W) {
      const int n = i / adj::kPassFields, f = i % adj::kPassFields;
      const int np = min(tp.i[L.npass + n], adj::kMaxPasses);
      if (k < np) dd[L.passes + static_cast<std::size_t>(poff[n] + k) * adj::kPassFields + f] = tp.pass(n, k)[f];
      more = more || k + 1 < np;
    }
    if (!__any_sync(0xffffffffu, more)) break;
  }
  const std::size_t bytes = record_bytes(L, nn, poff[nn]);
  T.sync();
  return bytes;
}

// A packed record in memory as a tape.
__device__ __forceinline__ adj::Tape packed_tape(unsigned char* rec, const adj::TapeLayout& L, int nn) {
  adj::Tape t;
  t.i = reinterpret_cast<std::int32_t*>(rec);
  t.d = reinterpret_cast<double*>(rec + record_ints_bytes(L, nn));
  t.L = L;
  t.first = t.i + L.ints;
  return t;
}

// Starts copying a record of `bytes` (global, 16-byte aligned, as is its size) into shared memory: 16-byte asynchronous
// copies spread over the team. copies_done, then a team barrier, make it visible.
template <int W>
__device__ __forceinline__ void copy_record(const unsigned char* src, int bytes, unsigned char* dst, const Team<W>& T) {
  const auto to = static_cast<unsigned>(__cvta_generic_to_shared(dst));
#pragma unroll 1
  for (int k = T.rank * 16; k < bytes; k += 32 * W * 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + k), "l"(src + k) : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The step's inputs into its tape, before the step: the scalars and every node's state, pass counts cleared.
template <int W>
__device__ __forceinline__ void tape_inputs(const adj::Tape& tp, const SimRegs& R, const Slot& S, int nn, const Team<W>& T) {
  const adj::TapeLayout& L = tp.L;
  if (T.leader()) {
    tp.d[L.scal] = R.t; tp.d[L.scal + 1] = R.zO; tp.d[L.scal + 2] = R.pitch; tp.d[L.scal + 3] = R.roll;
    tp.d[L.scal + 4] = R.vz; tp.d[L.scal + 5] = R.wth; tp.d[L.scal + 6] = R.wph;
  }
  for (int n = T.rank; n < nn; n += 32 * W) {
    tp.d[L.volIn + n] = S.vol[n]; tp.d[L.levelIn + n] = S.level[n];
    tp.d[L.cxIn + n] = S.cx[n]; tp.d[L.cyIn + n] = S.cy[n]; tp.d[L.czIn + n] = S.cz[n];
    tp.i[L.npass + n] = 0;
  }
  T.sync();
}

// The ring: a record at virtual offset v sits at v mod cap; a record that would run past the end starts the next lap
// instead. After the last write at virtual end E the ring holds exactly the records at offsets >= E - cap.
__device__ __forceinline__ long long ring_place(long long v, std::size_t cap, std::size_t maxRecord) {
  const long long c = static_cast<long long>(cap);
  if (v % c + static_cast<long long>(maxRecord) > c) v = (v / c + 1) * c;
  return v;
}

__device__ __forceinline__ long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return static_cast<long long>(t);
}

// The objective's adjoint at the state with scalars (zO, pitch, roll): every thread adds the same values.
__device__ __forceinline__ void add_sample_adjoint(const DevModel& M, double zO, double th, double ph, double aTrim, double aHeave, double* aSc) {
  const PoseD F = adj::pose_of(M, zO, th, ph);
  AdjPose aP;
  adj::zero(aP);
  adj::trim_heave_reverse(M, aTrim, aHeave, aP, aSc[1]);
  adj::pose_reverse(M, F, aP, aSc[0], aSc[1], aSc[2]);
}

// Sample k of the objective at state s with pose F: its values, their residuals into J, and where it was taken.
__device__ __forceinline__ void add_sample(const DevModel& M, const Pose& F, double pitch, const AdjRun& B, int inst, int k, long long s,
                                           const double* trimT, const double* heaveT, double& J, double* sampleS, bool leader) {
  double tr, hv;
  adj::trim_heave(M, PoseD{F.R00, F.R01, F.R02, F.R10, F.R11, F.R12, F.R20, F.R21, F.R22, F.tx, F.ty, F.tz, F.cth, F.iR}, pitch, tr, hv);
  J += (tr - trimT[k]) * (tr - trimT[k]) + (hv - heaveT[k]) * (hv - heaveT[k]);
  if (leader) {
    B.trim[static_cast<std::size_t>(inst) * B.nsamples + k] = tr; B.heave[static_cast<std::size_t>(inst) * B.nsamples + k] = hv;
    sampleS[k] = static_cast<double>(s);
  }
}

// 16 warps per SM in all: 128 registers a thread (left to itself the compiler takes 208 for 8-warp teams, and one fits an SM)
template <int W>
__global__ void __launch_bounds__(W * 32, 16 / W) adjoint_batch(const __grid_constant__ DevModel M, const __grid_constant__ AdjRun B, const __grid_constant__ SlotLayout SL,
                                                       const __grid_constant__ AdjLayout AL) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int team = blockIdx.x;
  Team<W> T;
  T.warp = threadIdx.x >> 5;
  T.lane = threadIdx.x & 31;
  T.rank = threadIdx.x;
  T.bar = 1;
  AdjTeam<W> AT{T.rank, 32 * W, T.warp, W, T.lane, 32, 1};
  Slot S = carve_slot(smem, SL);
  AdjSmem A = carve_adjoint(smem + SL.bytes, AL);
  const adj::TapeLayout TL = adj::tape_layout(M.nn, M.ng);
  const std::size_t recMax = record_bytes(TL, M.nn, M.nn * adj::kMaxPasses);
  const std::size_t recSize = 7 + 5 * static_cast<std::size_t>(M.nn);
  double* const ckpt = B.ckpt + static_cast<std::size_t>(team) * B.maxCkpt * recSize;
  unsigned char* const ring = B.arena + static_cast<std::size_t>(team) * B.arenaBytes;
  long long* const off = B.stepOff + static_cast<std::size_t>(team) * (B.maxSteps + 1);
  std::int32_t* const rb = B.recBytes + static_cast<std::size_t>(team) * (B.maxSteps + 1);
  double* const sink = B.sink + static_cast<std::size_t>(team) * (M.evCap + M.nmon + M.nmark + 1);
  std::int32_t* const isink = B.isink + static_cast<std::size_t>(team) * (M.evCap + 1);
  const adj::Tape sp = adj::tape_at(A.tape, TL);
  const int NS = B.nsamples;
  for (;;) {
    if (T.leader()) {
      const int q = atomicAdd(B.queue, 1);
      S.misc[kMiscInstance] = B.order == nullptr || q >= B.count ? q : B.order[q];
      S.misc[kMiscTaken] = W * (32 / kLevelLanes<false, W>);  // the level solve's list counter for the first step (team_step resets it)
    }
    T.sync();
    const int inst = S.misc[kMiscInstance];
    T.sync();
    if (inst >= B.count) return;
    const long long tStart = global_ns();
    long long tForward = 0, tRecompute = 0, tReverse = 0, nRecomputed = 0;
    const std::size_t ic = static_cast<std::size_t>(inst) * M.nc;
    const AdjInst I{B.en + ic, B.area + ic, B.tOn + ic, sink, isink, M.nmon};
    // the event bookkeeping sinks: overflow and mark times set (nothing fires), so events never write
    for (int k = T.rank; k < M.nmon + M.nmark + 1; k += 32 * W) sink[k] = 1.0;
    SimRegs R;
    {
      // the instance's initial state
      const std::size_t in = static_cast<std::size_t>(inst) * M.nn;
      double* c = ckpt;  // checkpoint 0 is the initial state
      if (T.leader())
        for (int k = 0; k < 7; ++k) c[k] = B.st0[static_cast<std::size_t>(inst) * 7 + k];
      for (int n = T.rank; n < M.nn; n += 32 * W) {
        c[7 + n] = B.vol0[in + n]; c[7 + M.nn + n] = B.level0[in + n];
        c[7 + 2 * M.nn + n] = B.cx0[in + n]; c[7 + 3 * M.nn + n] = B.cy0[in + n]; c[7 + 4 * M.nn + n] = B.cz0[in + n];
      }
      __threadfence_block();
      T.sync();
    }
    const double* trimT = B.trimT + static_cast<std::size_t>(inst) * NS;
    const double* heaveT = B.heaveT + static_cast<std::size_t>(inst) * NS;
    double J = 0;
    double aSc[6] = {0, 0, 0, 0, 0, 0};
    int k = 0, err = 0;
    long long S_end = 0, kept = 0;
    // stretch g = -1: forward from the initial state with checkpoints, the objective's samples and (tapeForward) every
    // step's record; then the segments, last first: one whose records the ring no longer holds is stepped again from its
    // checkpoint into the ring (every later segment has been reversed already, so the whole ring is free; it holds K
    // records of the largest size), and each is reversed. Both kinds of stretch run through one call of the step, of
    // which three inlined copies and the reverse did not fit the instruction caches.
    for (long long g = -1;;) {
      const bool forward = g < 0;
      const long long s0 = forward ? 0 : g * B.K;
      const long long s1 = forward ? B.maxSteps : (s0 + B.K < S_end ? s0 + B.K : S_end);
      const long long tSeg = global_ns();
      if (forward || !(B.tapeForward && off[s0] >= kept)) {
        load_state(ckpt + static_cast<std::size_t>(forward ? 0 : g) * recSize, R, S, M, T);
        *S.pose = make_pose(M, R.zO, R.pitch, R.roll);
        park(S.parked, R);
        T.sync();
        const bool record = !forward || B.tapeForward;
        long long s = s0, v = 0;
        for (;; ++s) {
          if (forward) {
            if (s % B.K == 0 && s > 0) {
              save_state(ckpt + static_cast<std::size_t>(s / B.K) * recSize, R, S, M.nn, T);
              T.sync();
            }
            if (R.foundered || R.t >= B.tMax) break;
          }
          if (s >= s1) break;
          while (forward && k < NS && R.t >= B.sampleT[k]) {
            add_sample(M, *S.pose, R.pitch, B, inst, k, s, trimT, heaveT, J, A.sampleS, T.leader());
            ++k;
          }
          if (record) tape_inputs(sp, R, S, M.nn, T);
          team_step<false, W>(M, R, S, I, T, GpuTape{sp, record});
          if (record) {
            T.sync();
            v = ring_place(v, B.arenaBytes, recMax);
            if (T.leader()) off[s] = v;
            const std::size_t bytes = store_record(sp, M.nn, A.poff, ring + v % static_cast<long long>(B.arenaBytes), T);
            if (T.leader()) rb[s] = static_cast<std::int32_t>(bytes);
            v += static_cast<long long>(bytes);
          }
        }
        if (forward) {
          S_end = s;
          // the ring holds the records at virtual offsets >= v - cap: a segment is reversed from the ring when its first
          // step's record is among them
          kept = B.tapeForward ? v - static_cast<long long>(B.arenaBytes) : LLONG_MAX;
        } else {
          nRecomputed += s1 - s0;
        }
      }
      if (forward) {
        for (; k < NS; ++k) add_sample(M, *S.pose, R.pitch, B, inst, k, S_end, trimT, heaveT, J, A.sampleS, T.leader());
        const double zE = R.zO, thE = R.pitch, phE = R.roll;
        __threadfence_block();
        T.sync();
        tForward = global_ns() - tStart;
        for (int n = T.rank; n < M.nn; n += 32 * W) { A.as.aVol[n] = 0; A.as.aLevel[n] = 0; A.as.aCx[n] = 0; A.as.aCy[n] = 0; A.as.aCz[n] = 0; }
        for (int c = T.rank; c < M.nc; c += 32 * W) A.grad[c] = 0;
        T.sync();
        // the samples at the final state (the objective's values of the trim and heave, recomputed from the outputs)
        for (int q = 0; q < NS; ++q)
          if (static_cast<long long>(A.sampleS[q]) == S_end) {
            const double tr = B.trim[static_cast<std::size_t>(inst) * NS + q], hv = B.heave[static_cast<std::size_t>(inst) * NS + q];
            add_sample_adjoint(M, zE, thE, phE, 2 * (tr - trimT[q]), 2 * (hv - heaveT[q]), aSc);
          }
        g = (S_end + B.K - 1) / B.K - 1;
        if (g < 0) break;
        continue;
      }
      __threadfence_block();
      T.sync();
      const long long tRev = global_ns();
      tRecompute += tRev - tSeg;
      // the record of step st is reversed where it was copied: into the tape's place, or (stageRecords) by turns there and
      // into the raw buffer, each while the step after it is reversed
      unsigned char* here = A.tape;
      copy_record(ring + off[s1 - 1] % static_cast<long long>(B.arenaBytes), rb[s1 - 1], here, T);
      for (long long st = s1 - 1; st >= s0; --st) {
        copies_done();
        T.sync();
        const adj::Tape tp = packed_tape(here, TL, M.nn);
        if (st > s0) {
          const unsigned char* next = ring + off[st - 1] % static_cast<long long>(B.arenaBytes);
          if (B.stageRecords) {
            here = here == A.tape ? A.raw : A.tape;
            copy_record(next, rb[st - 1], here, T);
          } else if (T.leader()) {
            // or at least into L2
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(next), "r"(static_cast<unsigned>(rb[st - 1])) : "memory");
          }
        }
        adj::reverse_step(AT, M, tp, I.en(), I.area(), I.tOn(), A.rs, A.as, aSc, A.grad, &err);
        for (int q = 0; q < NS; ++q)
          if (static_cast<long long>(A.sampleS[q]) == st) {
            const double tr = B.trim[static_cast<std::size_t>(inst) * NS + q], hv = B.heave[static_cast<std::size_t>(inst) * NS + q];
            add_sample_adjoint(M, tp.d[TL.scal + 1], tp.d[TL.scal + 2], tp.d[TL.scal + 3], 2 * (tr - trimT[q]), 2 * (hv - heaveT[q]), aSc);
          }
        T.sync();
        if (!B.stageRecords && st > s0) copy_record(ring + off[st - 1] % static_cast<long long>(B.arenaBytes), rb[st - 1], here, T);
      }
      tReverse += global_ns() - tRev;
      if (--g < 0) break;
    }
    T.sync();
    for (int c = T.rank; c < M.nc; c += 32 * W) B.grad[ic + c] = A.grad[c];
    if (err) atomicOr(B.error + inst, err);
    if (T.leader()) {
      B.J[inst] = J; B.steps[inst] = S_end;
      B.phaseNs[3 * static_cast<std::size_t>(inst)] = tForward;
      B.phaseNs[3 * static_cast<std::size_t>(inst) + 1] = tRecompute;
      B.phaseNs[3 * static_cast<std::size_t>(inst) + 2] = tReverse;
      B.recomputed[inst] = nRecomputed;
    }
    T.sync();
  }
}

}  // namespace

std::size_t adjoint_tape_bytes(int nn, int ng) { return record_bytes(adj::tape_layout(nn, ng), nn, nn * adj::kMaxPasses); }
std::size_t adjoint_record_bytes(int nn, int ng, int passRecords) { return record_bytes(adj::tape_layout(nn, ng), nn, passRecords); }

cudaError_t configure_adjoint_kernel(int W, std::size_t smem) {
  const int b = static_cast<int>(smem);
  switch (W) {
    case 4: return cudaFuncSetAttribute(adjoint_batch<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    case 8: return cudaFuncSetAttribute(adjoint_batch<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    case 16: return cudaFuncSetAttribute(adjoint_batch<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  }
  return cudaErrorInvalidValue;
}

cudaError_t adjoint_occupancy(int W, std::size_t smem, int* blocksPerSM) {
  switch (W) {
    case 4: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocksPerSM, adjoint_batch<4>, 4 * 32, smem);
    case 8: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocksPerSM, adjoint_batch<8>, 8 * 32, smem);
    case 16: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocksPerSM, adjoint_batch<16>, 16 * 32, smem);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_adjoint_kernel(int W, const DevModel& M, const AdjRun& B, const SlotLayout& SL, const AdjLayout& AL, int teams,
                                  cudaStream_t stream) {
  const std::size_t smem = static_cast<std::size_t>(SL.bytes) + AL.bytes;
  switch (W) {
    case 4: adjoint_batch<4><<<teams, 4 * 32, smem, stream>>>(M, B, SL, AL); break;
    case 8: adjoint_batch<8><<<teams, 8 * 32, smem, stream>>>(M, B, SL, AL); break;
    case 16: adjoint_batch<16><<<teams, 16 * 32, smem, stream>>>(M, B, SL, AL); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace ssb
