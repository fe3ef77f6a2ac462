// One time step of one simulation, computed by a team of W warps (W = 1, 2, 4, 8 or 16). The physics is the reference's
// kernel::step in the "portable" (double precision) and "portable32" (single-precision column partials) numerics
// (engine/include/sinksim/kernel/step.hpp:41-54), reproduced bit for bit:
//
//   * the buoyancy integral keeps the reference's 256 partial sums (partial p sums columns p, p+256, ... in
//     order), reduces each group of 32 partials with the halving tree (offsets 16..1) and adds the eight group
//     results in order (kernel/reduce.hpp:12-79, hydro.hpp:241-258). The team's warps share the eight groups: lane l
//     holds partial w*32+l of group w, and a shuffle butterfly performs the tree;
//   * a node pass keeps the reference's 32 lane partials over strided segments and the same tree
//     (hydro.hpp:305-316, reduce.hpp:52-71), except the lowest and highest point, which have the same bits however they
//     are found (extents.h); a group of kLevelLanes lanes forms them, each lane combining several
//     tree lanes' partials in the tree's order before the shuffles, so a warp solves 32 / kLevelLanes groups at once;
//   * every other reduction (group sums, incidence gathers, sea inflow, excess, loads, monitors, water) runs in
//     the reference's serial order, and every expression keeps its operation order (no contraction: -fmad=false).
//     The one count that is not a floating-point sum, a node's degree, is formed with shared-memory atomics.
//
// Every thread of the team holds identical copies of the scalars it uses, so control flow stays uniform; the team's
// threads wait on one another only at the team barrier (Team::sync: __syncwarp for one warp, a named barrier for
// more) between phases that exchange per-node or per-connection arrays through shared memory.
#pragma once

#include <cstdint>

#include "device_model.h"
#include "portable_math.cuh"
#include "scheme.h"

namespace ssb {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kLanes = 32;

// What a step issues must come from the instruction caches: with everything inlined and unrolled the kernel was 396 KB
// of code, and once the level solve issued a third of its instructions the warps waited for code most of the time (8.8 of
// 15.8 warps per issue, 1-warp teams). So the portable math, the extremes and the buoyancy are called, and loops that need
// no overlap are not unrolled: 152 to 155 KB in double precision and 138 to 141 in single precision, half of it outside the
// step. When that came, together with the sums a lane per column and one warp for the motion (move_body), on B200: 2,048
// uneven titanic64 runs to 20 min 371 ms against 469, a fleet of 96 ships to 5 min 36.5 against 62.4, one run to 5 min 29.1
// against 32.2, 48 portable32 runs to 15 min 68 against 83. At 128 registers a thread (16 warps an SM) the double precision
// kernels spill 68 to 192 bytes and the fleets' up to 192; what a build spills does not order its times.
static __device__ __noinline__ double2 trig_of(double x) {
  double s, c;
  pm::sin_cos(x, s, c);
  return double2{s, c};
}
static __device__ __noinline__ double pow_of(double x, double y) { return pm::pow(x, y); }

// The pose of (zO, pitch th, roll ph); a whole warp calls it (even lanes take the pitch's sine and cosine, odd lanes the
// roll's, and they swap).
__device__ __forceinline__ Pose make_pose(const DevModel& M, double zO, double th, double ph) {
  const bool odd = threadIdx.x & 1;
  const double2 t = trig_of(odd ? ph : th);
  const double os = __shfl_xor_sync(kFull, t.x, 1), oc = __shfl_xor_sync(kFull, t.y, 1);
  const double sth = odd ? os : t.x, cth = odd ? oc : t.y, sph = odd ? t.x : os, cph = odd ? t.y : oc;
  Pose F;
  F.R00 = cth; F.R01 = sth * sph; F.R02 = sth * cph;
  F.R10 = 0;   F.R11 = cph;       F.R12 = -sph;
  F.R20 = -sth; F.R21 = cth * sph; F.R22 = cth * cph;
  F.tx = M.XO - (F.R00 * M.g0x + F.R01 * M.g0y + F.R02 * M.g0z);
  F.ty = M.YO - (F.R10 * M.g0x + F.R11 * M.g0y + F.R12 * M.g0z);
  F.tz = zO - (F.R20 * M.g0x + F.R21 * M.g0y + F.R22 * M.g0z);
  F.cth = cth;
  F.iR = 1 / F.R22;
  F.fR20 = static_cast<float>(F.R20);
  F.fR21 = static_cast<float>(F.R21);
  F.fR22 = static_cast<float>(F.R22);
  F.ftz = static_cast<float>(F.tz);
  F.fiR = 1.0f / F.fR22;
  return F;
}

__device__ __forceinline__ double world_z(const Pose& F, double x, double y, double z) {
  return F.R20 * x + F.R21 * y + F.R22 * z + F.tz;
}

// ----------------------------------------------------------------------------- butterfly steps of the canonical tree
// At offset `off` the tree combines partial l (l < off) with partial l + off. With xor shuffles every lane pairs
// with lane ^ off; sums are exact to swap (IEEE addition is commutative), so every lane ends with the bits of the tree's
// lane 0.

template <class T>
__device__ __forceinline__ T bsum(T v, int off, unsigned mask = kFull) { return v + __shfl_xor_sync(mask, v, off); }

// ----------------------------------------------------------------------------- a team of W warps stepping one simulation

// Thread `rank` of the team (0 .. 32 W - 1), its warp and lane. Teams of more than one warp synchronise on their own
// named barrier (ids 1..15; 0 is __syncthreads), so teams in one block never wait on each other.
template <int W>
struct Team {
  int rank, warp, lane, bar;
  __device__ __forceinline__ void sync() const {
    if constexpr (W == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(W * 32) : "memory");
  }
  __device__ __forceinline__ bool leader() const { return rank == 0; }
};

// ----------------------------------------------------------------------------- world extents

// The lowest bottom (MAX false) or highest top (MAX true) of set n in the world: a node's segments, or the hull's
// columns for n == M.nn (tops only). Scanned over the set's extent list for the signs of R20 and R21 (extents.h: the
// same bits as over the whole set, for 4 to 10 points instead of 136), by `lanes` threads, this one taking every
// lanes-th point from `sub`; the caller combines them. An attitude beyond a quarter turn (R22 < 0, only from a restored
// state: the step clamps pitch and roll) scans the whole set.
template <bool MIXED>
struct Prec;
template <>
struct Prec<false> {
  using T = double;
  using V2 = double2;
  static __device__ __forceinline__ const V2* exXY(const DevModel& M) { return M.exXY; }
  static __device__ __forceinline__ const T* exZ(const DevModel& M) { return M.exZ; }
  static __device__ __forceinline__ const V2* segXY(const DevModel& M) { return M.segXY; }
  static __device__ __forceinline__ const V2* segLH(const DevModel& M) { return M.segLH; }
  static __device__ __forceinline__ const T* segAr(const DevModel& M) { return M.segAr; }
  static __device__ __forceinline__ const V2* colXY(const DevModel& M) { return M.colXY; }
  static __device__ __forceinline__ const V2* colLH(const DevModel& M) { return M.colLH; }
  static __device__ __forceinline__ const T* colAr(const DevModel& M) { return M.colA; }
  static __device__ __forceinline__ T R20(const Pose& F) { return F.R20; }
  static __device__ __forceinline__ T R21(const Pose& F) { return F.R21; }
  static __device__ __forceinline__ T R22(const Pose& F) { return F.R22; }
  static __device__ __forceinline__ T tz(const Pose& F) { return F.tz; }
  static __device__ __forceinline__ T iR(const Pose& F) { return F.iR; }
};
template <>
struct Prec<true> {
  using T = float;
  using V2 = float2;
  static __device__ __forceinline__ const V2* exXY(const DevModel& M) { return M.exXYf; }
  static __device__ __forceinline__ const T* exZ(const DevModel& M) { return M.exZf; }
  static __device__ __forceinline__ const V2* segXY(const DevModel& M) { return M.segXYf; }
  static __device__ __forceinline__ const V2* segLH(const DevModel& M) { return M.segLHf; }
  static __device__ __forceinline__ const T* segAr(const DevModel& M) { return M.segArf; }
  static __device__ __forceinline__ const V2* colXY(const DevModel& M) { return M.colXYf; }
  static __device__ __forceinline__ const V2* colLH(const DevModel& M) { return M.colLHf; }
  static __device__ __forceinline__ const T* colAr(const DevModel& M) { return M.colAf; }
  static __device__ __forceinline__ T R20(const Pose& F) { return F.fR20; }
  static __device__ __forceinline__ T R21(const Pose& F) { return F.fR21; }
  static __device__ __forceinline__ T R22(const Pose& F) { return F.fR22; }
  static __device__ __forceinline__ T tz(const Pose& F) { return F.ftz; }
  static __device__ __forceinline__ T iR(const Pose& F) { return F.fiR; }
};

// With `first` only the first point of this thread is looked at, and `whole` is cleared when the list has more than the
// threads' first ones.
template <bool MIXED>
__device__ __noinline__ typename Prec<MIXED>::T scan_extreme(const DevModel& M, const Pose& F, int n, bool top, int sub, int lanes, bool first,
                                                              bool& whole) {
  using P = Prec<MIXED>;
  using T = typename P::T;
  const T R20 = P::R20(F), R21 = P::R21(F), R22 = P::R22(F), tz = P::tz(F);
  const typename P::V2* xy = P::exXY(M);
  const T* z = P::exZ(M);
  int j, end, zs = 1;
  if (F.R22 >= 0) {
    const int list = ((F.R20 < 0 ? 2 : 0) + (F.R21 < 0 ? 4 : 0) + (top ? 1 : 0)) * (M.nn + 1) + n;
    j = __ldg(M.exStart + list);
    end = __ldg(M.exStart + list + 1);
  } else {
    const bool hull = n == M.nn;
    xy = hull ? P::colXY(M) : P::segXY(M);
    z = reinterpret_cast<const T*>(hull ? P::colLH(M) : P::segLH(M)) + (top ? 1 : 0);
    zs = 2;
    j = hull ? 0 : __ldg(M.segStart + n);
    end = j + (hull ? M.ncol : __ldg(M.segCount + n));
  }
  whole = !first || end - j <= lanes;
  if (!whole) end = j + lanes;
  T best = top ? T(-1e9) : T(1e9);
#pragma unroll 2
  for (j += sub; j < end; j += lanes) {
    const auto p = __ldg(xy + j);
    const T w = R20 * p.x + R21 * p.y + tz + R22 * __ldg(z + static_cast<std::size_t>(j) * zs);
    if (top ? w > best : w < best) best = w;
  }
  return best;
}

template <bool MIXED>
__device__ __forceinline__ typename Prec<MIXED>::T node_extreme(const DevModel& M, const Pose& F, int n, bool top, int sub, int lanes) {
  bool whole;
  return scan_extreme<MIXED>(M, F, n, top, sub, lanes, false, whole);
}

// ----------------------------------------------------------------------------- buoyancy (hydro pass, tree order)

// One column into a buoyancy partial (kernel/reduce.hpp:39-49 in double, :131-142 in float): the same expressions in
// the same order for T = double (portable) and T = float (portable32). The hull's highest point is not formed here but
// from the columns' extent list (node_extreme: 24 to 41 points on titanic64 for 4,408), and a dry column adds zeros,
// which leaves every sum as it is. The loop is bound by the instructions it issues; with both out of it, on B200:
// 2,048 uneven titanic64 runs to 20 min 493 ms against 512, a fleet of 96 ships to 5 min 63.6 against 68.7, one run to
// 5 min 33.4 against 35.1.
template <class T>
struct ColPartial {
  T V, Mx, My, Mz;
};

template <class T>
__device__ __forceinline__ void clip_column(T x, T y, T lo, T hi, T A, T R20, T R21, T tz, T iR, ColPartial<T>& p) {
  const T base = R20 * x + R21 * y + tz;
  const T zp = -base * iR;
  const T s = zp <= lo ? T(0) : (zp >= hi ? hi - lo : zp - lo);
  const T v = A * s;
  p.V += v; p.Mx += v * x; p.My += v * y; p.Mz += v * (lo + T(0.5) * s);
}

// One segment into a node-pass partial (kernel/reduce.hpp:52-71 in double, :144-164 in float) without the pass's world
// extent, which comes from the extent lists (node_extreme). A dry segment adds zeros, which leaves every sum as it is
// (a sum is never -0), so the lanes of a warp stay together.
template <class T>
struct SegPartial {
  T vol, dv, mx, my, mz;
};

template <class T>
__device__ __forceinline__ void clip_segment(T x, T y, T a, T b, T A, T R20, T R21, T tz, T iR, T h, SegPartial<T>& p) {
  const T base = R20 * x + R21 * y + tz;
  const T zp = (h - base) * iR;
  const bool dry = zp <= a, full = zp >= b;
  const T L = dry ? T(0) : (full ? b - a : zp - a);
  const T v = A * L;
  p.dv += (dry || full) ? T(0) : A;
  p.vol += v; p.mx += v * x; p.my += v * y; p.mz += v * (a + T(0.5) * L);
}

template <class T> struct Vec2;
template <> struct Vec2<double> { using type = double2; };
template <> struct Vec2<float> { using type = float2; };

// A load of the column table: from shared memory (kStaged: the table staged there), or through the read-only data cache
// from global memory; kStreamed: without a place in L1, which a lone simulation's step would sweep clean with the 176 KB
// it reads once, while the segments and the small tables are read again.
enum ColumnSource { kCached, kStreamed, kStaged };

__device__ __forceinline__ double2 load_streamed(const double2* p) {
  double2 v;
  asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ double load_streamed(const double* p) {
  double v;
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 load_streamed(const float2* p) {
  float2 v;
  asm("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float load_streamed(const float* p) {
  float v;
  asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

template <ColumnSource SRC, class P>
__device__ __forceinline__ P load_col(const P* p) {
  if constexpr (SRC == kStaged) return *p;
  else if constexpr (SRC == kStreamed) return load_streamed(p);
  else return __ldg(p);
}

// Lane `lane`'s partial of tree w: columns w*32 + lane + 256 k in increasing k, AT_ONCE at a time (the loads of
// all issue before the first is clipped; the clips stay in order). Teams of 8 and 16 warps wait for the loads: they take
// four, past L1. Smaller ones share an SM with others that fill the wait and that read the same columns from L1, and two
// need less code and pad less. On B200: 16 warps, one run to 5 min 21.7 ms, cached 25.8; 8 warps, 250 titanic64 runs to 1 min
// 4.11, cached in twos 4.54 (portable32 3.50, 3.46); 4 warps, 500 runs to 5 min 38.3, past L1 in fours 39.9 (portable32, 401
// runs to 61 s 4.72, 5.02).
template <class T, ColumnSource SRC, int AT_ONCE>
__device__ __forceinline__ ColPartial<T> column_partial(const typename Vec2<T>::type* xy, const typename Vec2<T>::type* lh, const T* area,
                                                        int ncol, int first, T R20, T R21, T tz, T iR) {
  ColPartial<T> p{T(0), T(0), T(0), T(0)};
#pragma unroll 1
  for (int i = first; i < ncol; i += AT_ONCE * 256) {
    typename Vec2<T>::type a[AT_ONCE], b[AT_ONCE];
    T A[AT_ONCE];
#pragma unroll
    for (int k = 0; k < AT_ONCE; ++k) {
      // past the table's end: the last column read again with no footprint, which adds zeros
      const int j = i + 256 * k < ncol ? i + 256 * k : i;
      a[k] = load_col<SRC>(xy + j);
      b[k] = load_col<SRC>(lh + j);
      A[k] = i + 256 * k < ncol ? load_col<SRC>(area + j) : T(0);
    }
#pragma unroll
    for (int k = 0; k < AT_ONCE; ++k) clip_column<T>(a[k].x, a[k].y, b[k].x, b[k].y, A[k], R20, R21, tz, iR, p);
  }
  return p;
}

// The column table staged in shared memory (stage_columns): (x, y) pairs, (zlo, zhi) pairs and footprints of every
// column, in the arithmetic's type, each array at a 16-byte boundary.
template <class T>
struct StagedColumns {
  std::size_t xy, lh, area, bytes;
};

template <class T>
__host__ __device__ __forceinline__ StagedColumns<T> staged_columns(int ncol) {
  using V2 = typename Vec2<T>::type;
  StagedColumns<T> c;
  const std::size_t n = static_cast<std::size_t>(ncol);
  auto up16 = [](std::size_t b) { return (b + 15) & ~static_cast<std::size_t>(15); };
  c.xy = 0;
  c.lh = up16(n * sizeof(V2));
  c.area = c.lh + up16(n * sizeof(V2));
  c.bytes = c.area + up16(n * sizeof(T));
  return c;
}

// The eight trees are spread over the team's warps (warp v computes trees v, v + W, ...), and the last warp finds the
// hull's highest point; the results meet in shared memory (four values per tree, then the top) and every thread adds
// them in the reference's order (trees 0..7).
template <bool MIXED, int W>
__device__ __noinline__ void buoyancy_trees(const DevModel& M, const Pose& F, int warp, int lane, double* trees, const unsigned char* cols) {
  using P = Prec<MIXED>;
  using R = typename P::T;
#pragma unroll 1
  for (int w = warp; w < 8; w += W) {
    ColPartial<R> p;
    if (cols) {
      const StagedColumns<R> c = staged_columns<R>(M.ncol);
      p = column_partial<R, kStaged, 2>(reinterpret_cast<const typename P::V2*>(cols + c.xy), reinterpret_cast<const typename P::V2*>(cols + c.lh),
                                  reinterpret_cast<const R*>(cols + c.area), M.ncol, w * kLanes + lane, P::R20(F), P::R21(F), P::tz(F), P::iR(F));
    } else {
      p = column_partial<R, (W >= 8 ? kStreamed : kCached), (W >= 8 ? 4 : 2)>(P::colXY(M), P::colLH(M), P::colAr(M), M.ncol, w * kLanes + lane, P::R20(F), P::R21(F), P::tz(F), P::iR(F));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      p.V = bsum(p.V, off); p.Mx = bsum(p.Mx, off); p.My = bsum(p.My, off); p.Mz = bsum(p.Mz, off);
    }
    if (lane == 0) {
      double* t = trees + 4 * w;
      t[0] = p.V; t[1] = p.Mx; t[2] = p.My; t[3] = p.Mz;
    }
  }
  if (warp == W - 1) {
    R top = node_extreme<MIXED>(M, F, M.nn, true, lane, kLanes);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const R o = __shfl_xor_sync(kFull, top, off);
      if (o > top) top = o;
    }
    if (lane == 0) trees[32] = top;
  }
}

// The buoyancy result from the eight trees (after a team barrier that follows buoyancy_trees): every thread adds
// them in the reference's order and holds the same values.
__device__ __forceinline__ Buoy buoyancy_finish(const double* trees) {
  double V = trees[0], Mx = trees[1], My = trees[2], Mz = trees[3];
  for (int w = 1; w < 8; ++w) {
    const double* t = trees + 4 * w;
    V += t[0]; Mx += t[1]; My += t[2]; Mz += t[3];
  }
  Buoy b;
  b.V = V;
  b.x = V > 0 ? Mx / V : 0;
  b.y = V > 0 ? My / V : 0;
  b.z = V > 0 ? Mz / V : 0;
  b.top = trees[32];
  return b;
}

template <bool MIXED, int W>
__device__ __forceinline__ Buoy buoyancy(const DevModel& M, const Pose& F, const Team<W>& T, double* trees, const unsigned char* cols) {
  buoyancy_trees<MIXED, W>(M, F, T.warp, T.lane, trees, cols);
  T.sync();
  return buoyancy_finish(trees);
}

// ----------------------------------------------------------------------------- node pass (tree order)

struct PassR {
  double vol, dv, mx, my, mz;
};

// The kLevelLanes<MIXED, W> consecutive lanes of a warp that solve one group of nodes: `lane` is the lane in the warp, `sub` the
// lane in the group, `mask` the group's lanes.
struct LevelLanes {
  int lane, sub;
  unsigned mask;
};

template <bool MIXED, int W>
__device__ __forceinline__ LevelLanes level_lanes(int lane) {
  constexpr int LANES = kLevelLanes<MIXED, W>;
  return LevelLanes{lane, lane % LANES, (LANES == 32 ? kFull : (1u << (LANES & 31)) - 1u) << (lane / LANES * LANES)};
}

// The partials of two tree lanes 16 apart (first segments fa and fa + 16; PAIR), or of fa's tree lane alone, two of its
// segments per iteration, in one loop: each iteration takes the next segment of each, so the two accumulation chains run
// side by side; each keeps its own segments' order. A missing second segment is the first one again with no footprint,
// which adds zeros. AHEAD iterations' loads issue together.
template <class T, bool PAIR, int AHEAD>
__device__ __forceinline__ void segment_partials(const typename Vec2<T>::type* xy, const typename Vec2<T>::type* ab, const T* area, int fa,
                                                 int end, T R20, T R21, T tz, T iR, T h, SegPartial<T>& pa, SegPartial<T>& pb) {
  constexpr int kStep = PAIR ? kLanes : 2 * kLanes, kOff = PAIR ? kLanes / 2 : kLanes;
  pa = SegPartial<T>{T(0), T(0), T(0), T(0), T(0)};
  pb = pa;
#pragma unroll AHEAD
  for (int ja = fa; ja < end; ja += kStep) {
    const bool two = ja + kOff < end;
    const int jb = two ? ja + kOff : ja;
    const auto a0 = __ldg(xy + ja), b0 = __ldg(ab + ja), a1 = __ldg(xy + jb), b1 = __ldg(ab + jb);
    const T A0 = __ldg(area + ja), A1 = two ? __ldg(area + jb) : T(0);
    clip_segment<T>(a0.x, a0.y, b0.x, b0.y, A0, R20, R21, tz, iR, h, pa);
    clip_segment<T>(a1.x, a1.y, b1.x, b1.y, A1, R20, R21, tz, iR, h, PAIR ? pb : pa);
  }
}

// One level of the tree inside a lane: the lower tree lane's partial `lo` takes in the upper one's, with the operand
// order of the butterfly steps.
template <class T>
__device__ __forceinline__ void tree_pair(SegPartial<T>& lo, const SegPartial<T>& up) {
  lo.vol = lo.vol + up.vol; lo.dv = lo.dv + up.dv; lo.mx = lo.mx + up.mx; lo.my = lo.my + up.my; lo.mz = lo.mz + up.mz;
}

// The pass over a node's segments [s0, s1) with permeability mu at world level h: the 32 lane partials, the halving tree
// and the permeability scaling (hydro.hpp:295-316 / 338-349). Lane `sub` of a group of kLevelLanes lanes forms the partials
// of tree lanes sub + kLevelLanes j and combines them over the tree's upper levels (offsets 16 down to kLevelLanes) in
// registers; the lower levels are shuffles inside the group. Every lane of the group ends with the bits of tree lane 0.
// Every lane of the warp calls it (an empty range for a group without a node), so the groups' passes run side by side.
template <bool MIXED, int W>
__device__ __forceinline__ PassR node_pass(const DevModel& M, const Pose& F, int s0, int s1, double mu, double h, const LevelLanes& L) {
  using P = Prec<MIXED>;
  using T = typename P::T;
  constexpr int LANES = kLevelLanes<MIXED, W>;
  static_assert(LANES == 16 || LANES == 32, "a lane forms one or two of the tree's partials");
  constexpr int AHEAD = W >= 8 ? 2 : 1;  // large teams are bound by the loads' latency, small ones by issue slots
  const T hT = static_cast<T>(h);
  const int f = s0 + L.sub;
  const T R20 = P::R20(F), R21 = P::R21(F), tz = P::tz(F), iR = P::iR(F);
  const typename P::V2 *xy = P::segXY(M), *ab = P::segLH(M);
  const T* area = P::segAr(M);
  SegPartial<T> p, b;
  if constexpr (LANES == 32) {
    segment_partials<T, false, AHEAD>(xy, ab, area, f, s1, R20, R21, tz, iR, hT, p, b);
  } else {
    segment_partials<T, true, AHEAD>(xy, ab, area, f, s1, R20, R21, tz, iR, hT, p, b);  // tree lanes sub and sub + 16
    tree_pair(p, b);
  }
#pragma unroll
  for (int off = LANES / 2; off > 0; off >>= 1) {
    p.vol = bsum(p.vol, off); p.dv = bsum(p.dv, off); p.mx = bsum(p.mx, off);
    p.my = bsum(p.my, off); p.mz = bsum(p.mz, off);
  }
  PassR r;
  r.vol = static_cast<double>(p.vol) * mu;
  r.dv = static_cast<double>(p.dv) * mu * F.iR;
  r.mx = static_cast<double>(p.mx) * mu; r.my = static_cast<double>(p.my) * mu; r.mz = static_cast<double>(p.mz) * mu;
  return r;
}

// ----------------------------------------------------------------------------- per-warp view of the slot in shared memory

struct Slot {
  double *vol, *level, *cx, *cy, *cz, *area, *zmax, *hEff, *aEff, *tmp, *acc, *dV, *hydro;
  int* misc;
  PassR* passes;
  std::uint8_t* merged;
  std::uint8_t* dry;          // NodeFlag bits
  std::uint16_t* list;        // the groups the next level solve visits, misc[kMiscListed] of them (list_groups)
  std::uint8_t* wet;          // per 32 nodes, the flooded ones among them (their load terms)
  std::uint16_t* flow;        // the connections that can flow in this step (sort_connections)
  Pose* pose;                 // the current step's pose, and
  Pose* prev;                 // the last step's (that of the last level solve, between steps)
  Parked* parked;
  const unsigned char* cols;  // the column table staged in the block's shared memory, or null (read from global)
};

__device__ __forceinline__ Slot carve_slot(unsigned char* base, const SlotLayout& L) {
  Slot s;
  s.vol = reinterpret_cast<double*>(base + L.vol);
  s.level = reinterpret_cast<double*>(base + L.level);
  s.cx = reinterpret_cast<double*>(base + L.cx);
  s.cy = reinterpret_cast<double*>(base + L.cy);
  s.cz = reinterpret_cast<double*>(base + L.cz);
  s.area = reinterpret_cast<double*>(base + L.area);
  s.zmax = reinterpret_cast<double*>(base + L.zmax);
  s.hEff = reinterpret_cast<double*>(base + L.hEff);
  s.aEff = reinterpret_cast<double*>(base + L.aEff);
  s.acc = reinterpret_cast<double*>(base + L.acc);
  s.dV = reinterpret_cast<double*>(base + L.dV);
  s.tmp = reinterpret_cast<double*>(base + L.tmp);
  s.flow = reinterpret_cast<std::uint16_t*>(base + L.tmp);
  s.hydro = reinterpret_cast<double*>(base + L.hydro);
  s.misc = reinterpret_cast<int*>(base + L.misc);
  s.passes = reinterpret_cast<PassR*>(base + L.passes);
  s.merged = base + L.merged;
  s.dry = base + L.dry;
  s.wet = base + L.wet;
  s.list = reinterpret_cast<std::uint16_t*>(base + L.list);
  s.pose = reinterpret_cast<Pose*>(base + L.pose);
  s.prev = s.pose + 1;
  s.parked = reinterpret_cast<Parked*>(base + L.parked);
  s.cols = nullptr;
  return s;
}

// ----------------------------------------------------------------------------- free-surface levels (kernel/levels.hpp)
// What bounds the solve is the number of instructions a step issues, so it visits only the groups that hold water: at
// the end of a step one warp lists them (list_groups), and the lane groups of the team take them from the list. An
// empty node's level is its lowest segment bottom at the pose of the solve, which nothing reads before the node gets
// water or is written out; it is formed then (stale_level), from the pose kept for that. A listed unit (a merged group
// or one node) takes its world extent from the extent lists first, so the pass the reference makes only for the extent
// of a full node, or of one whose starting level lies outside it, is not made. Every pass of a warp's lane groups runs
// through one call site under a warp-wide loop: two half-warps in different solvers would otherwise issue everything
// twice. Centroids are divided node by node afterwards, a thread per node (team_step).
// Measured on B200 when it came, with the step as it then was: 2,048 titanic64 instances of the uneven batch to 20 min
// 512 ms (805 ms with a pass over every segment of every node, a divergent solver per half-warp and the extents in the
// pass), 264 liner runs to 15 min 119 ms (152), one titanic64 run to 5 min 35.1 ms (40.5). The first look at the extent
// lists, members side by side, list entries that carry the members, the pair's sharing in all lanes and the columns past
// L1 in large teams: 192 runs to 1 h 264 ms (353 before), one run 21.7 (29.1), 264 liner runs 95 (108), 2,048 uneven runs
// 348 (371).

// S.dry[n].
enum NodeFlag : std::uint8_t {
  kStale = 1,      // empty at the last level solve: S.level[n] is not formed yet
  kEmptyNode = 2,  // empty at the coming one
  kZeroVolume = 4, // ... in a merged group, which empties its members
  kSolved = 8,     // passes were made for it at this one
  kNoTop = 16      // ... without its highest point: S.zmax[n] is not formed
};

// Where a step's forward computation records what its reverse (the adjoint, adjoint_kernel.cu) needs: every unit's start
// (starting level and world extent), every node pass of the level solve (node, pass number within the node's solve,
// level, result) and the solved levels. kLazy: empty nodes are left out of the solve, their levels formed on demand.
// The batch kernels pass NoTape, whose hooks are empty and compile away.
struct NoTape {
  static constexpr bool kLazy = true;
  __device__ __forceinline__ void start(int, double, double, double, const LevelLanes&) const {}
  __device__ __forceinline__ void pass(int, int, double, const PassR&, const LevelLanes&) const {}
  template <int W>
  __device__ __forceinline__ void solved(const DevModel&, const Slot&, const Team<W>&) const {}
};

// Lists the groups the next level solve visits, in increasing order, and flags the nodes of the others; one warp calls
// it. A group is left out (kLazy) when neither its members nor their sum exceed the empty volume: then the solve would
// find it empty merged or not. A group of one is listed as its node, which is all the solve needs of it (its merged flag
// stays 0); a larger one as kListedGroup + its index, and its taker loads the entry made with the model. (The whole entry in
// the list, 8 bytes a group, kept hulls of few connections from fitting a block.)
constexpr int kListedGroup = 0x8000;

template <bool LAZY>
__device__ __forceinline__ void list_groups(const DevModel& M, Slot& S, int lane) {
  int count = 0;
#pragma unroll 1
  for (int g0 = 0; g0 < M.ng; g0 += kLanes) {
    const bool any = g0 + lane < M.ng;
    const int g = any ? g0 + lane : g0;
    const uint2 bits = __ldg(reinterpret_cast<const uint2*>(M.groupEntry) + g);
    const int n0 = bits.x & 0xffff, n1 = bits.x >> 16, N = bits.y & 0xff, mode = (bits.y >> 8) & 0xff;
    const double v0 = S.vol[n0], v1 = S.vol[n1];  // (n1 is n0 in a group of one)
    double V = v0;
    bool live = !LAZY || !(v0 <= kEmptyVolume);
    if (N >= 2) {
      V += v1;
      live = live || !(v1 <= kEmptyVolume);
    }
    if (N > 2) {
      const int* m = M.gNodes + __ldg(M.gStart + g);
      const int all = __ldg(M.gCount + g);
#pragma unroll 1
      for (int k = 2; k < all; ++k) {
        const double v = S.vol[__ldg(m + k)];
        V += v;
        live = live || !(v <= kEmptyVolume);
      }
    }
    live = any && (live || !(V <= kEmptyVolume));
    if (any && !live) {
      const bool merged = N >= 2 && mode == 1;
      const int flags = kEmptyNode | (merged ? kZeroVolume : 0);
      S.merged[g] = merged ? 1 : 0;
      S.dry[n0] |= flags;
      if (N >= 2) S.dry[n1] |= flags;
      if (N > 2) {
        const int* m = M.gNodes + __ldg(M.gStart + g);
        const int all = __ldg(M.gCount + g);
#pragma unroll 1
        for (int k = 2; k < all; ++k) S.dry[__ldg(m + k)] |= flags;
      }
    }
    const unsigned mask = __ballot_sync(kFull, live);
    if (live) S.list[count + __popc(mask & ((1u << lane) - 1u))] = static_cast<std::uint16_t>(N == 1 ? n0 : kListedGroup + g);
    count += __popc(mask);
  }
  if (lane == 0) S.misc[kMiscListed] = count;
}

// A group's combined value of node_extreme over its lanes.
template <bool MIXED, int W>
__device__ __forceinline__ double group_extreme(const DevModel& M, const Pose& F, int n, bool top, const LevelLanes& L) {
  constexpr int LANES = kLevelLanes<MIXED, W>;
  auto v = node_extreme<MIXED>(M, F, n, top, L.sub, LANES);
#pragma unroll
  for (int off = LANES / 2; off > 0; off >>= 1) {
    const auto o = __shfl_xor_sync(L.mask, v, off);
    if (top ? o > v : o < v) v = o;
  }
  return static_cast<double>(v);
}

// Node n's level as the last solve left it (an empty node's is formed here); one thread, or a lane group.
template <bool MIXED>
__device__ __forceinline__ double stale_level(const DevModel& M, const Slot& S, int n) {
  return (S.dry[n] & kStale) ? static_cast<double>(node_extreme<MIXED>(M, *S.prev, n, false, 0, 1)) : S.level[n];
}

template <bool MIXED, int W>
__device__ __forceinline__ double group_level(const DevModel& M, const Slot& S, int n, const LevelLanes& L) {
  return (S.dry[n] & kStale) ? group_extreme<MIXED, W>(M, *S.prev, n, false, L) : S.level[n];
}

// A first look at the world extents of one node, or of two side by side, by a lane group: z[0] and z[1] the lowest bottom
// and highest top of n0, z[2] and z[3] those of n1, over the first points of their lists. Each quarter of the lanes looks
// at one list (with one node, two quarters share each); `whole` says whether that was all of every list.
struct Extents {
  double z[4];
  bool whole;
};

template <bool MIXED, int W>
__device__ __forceinline__ Extents first_extents(const DevModel& M, const Pose& F, int n0, int n1, bool two, const LevelLanes& L) {
  constexpr int LANES = kLevelLanes<MIXED, W>, Q = LANES / 4;
  const int quarter = L.sub / Q, at = L.sub % Q;
  const bool top = quarter & 1;
  bool whole = true;
  auto v = scan_extreme<MIXED>(M, F, two && quarter >= 2 ? n1 : n0, top, two ? at : (quarter >> 1) * Q + at, two ? Q : 2 * Q, true, whole);
#pragma unroll
  for (int off = Q / 2; off > 0; off >>= 1) {
    const auto o = __shfl_xor_sync(L.mask, v, off);
    if (top ? o > v : o < v) v = o;
  }
  const auto o = __shfl_xor_sync(L.mask, v, 2 * Q);
  if (!two && (top ? o > v : o < v)) v = o;
  Extents e;
  const int base = L.lane - L.sub;
#pragma unroll
  for (int k = 0; k < 4; ++k) e.z[k] = static_cast<double>(__shfl_sync(L.mask, v, base + k * Q));
  e.whole = (__ballot_sync(L.mask, whole) & L.mask) == L.mask;
  return e;
}

// The solved values of a node whose last pass was p: the pass's sums go to scratch arrays that are dead until the heads,
// where the node's thread divides the centroid (set_centroid).
__device__ __forceinline__ void store_solved(Slot& S, int n, double level, double area, const PassR& p) {
  S.level[n] = level; S.area[n] = area;
  S.acc[n] = p.vol; S.hEff[n] = p.mx; S.aEff[n] = p.my; S.tmp[n] = p.mz;
}

__device__ __forceinline__ void set_centroid(Slot& S, int n) {
  const double vol = S.acc[n];
  if (vol > kCentroidMinVolume) { S.cx[n] = S.hEff[n] / vol; S.cy[n] = S.aEff[n] / vol; S.cz[n] = S.tmp[n] / vol; }
}

// The volumes and solved values of a merged group of N nodes after its Newton iteration (levels.hpp:113-162); P holds
// the members' last passes, V their water. One lane.
__device__ __forceinline__ void share_group(const DevModel& M, Slot& S, const PassR* P, const int* m, int N, double V, double h) {
  double tot = 0;
#pragma unroll 1
  for (int k = 0; k < N; ++k) tot += P[k].vol;
  double assigned = 0;
#pragma unroll 1
  for (int k = 0; k < N - 1; ++k) {
    const int n = __ldg(m + k);
    double v = tot > 0 ? V * P[k].vol / tot : V / static_cast<double>(N);
    const double vm = __ldg(M.vmax + n);
    if (v > vm) v = vm;
    S.vol[n] = v;
    assigned += v;
  }
  const double vmaxLast = __ldg(M.vmax + __ldg(m + N - 1));
  if (V - assigned > vmaxLast) {
    // the last member would overflow: the ones before it hold V - vmaxLast, filled from the end (levels.hpp:136-155)
    const double need = V - vmaxLast;
    double capped = 0;
#pragma unroll 1
    for (int k = N - 2; k >= 0; --k) {
      double prior = 0;
#pragma unroll 1
      for (int j = 0; j < k; ++j) prior += S.vol[__ldg(m + j)];
      const int n = __ldg(m + k);
      const double v = (need - capped) - prior;
      const double vm = __ldg(M.vmax + n);
      if (v > vm && k > 0) {
        S.vol[n] = vm;
        capped += vm;
        continue;
      }
      S.vol[n] = v;
      break;
    }
    assigned = 0;
#pragma unroll 1
    for (int k = 0; k < N - 1; ++k) assigned += S.vol[__ldg(m + k)];
  }
  S.vol[__ldg(m + N - 1)] = V - assigned;
#pragma unroll 1
  for (int k = 0; k < N; ++k) store_solved(S, __ldg(m + k), h, P[k].dv, P[k]);
}

// share_group for a group of two, by all lanes of its group: p0 the first member's pass, p1 the second's, tot their volume.
__device__ __forceinline__ void share_pair(Slot& S, const PassR& p0, const PassR& p1, int n0, int n1, double vmax0, double vmax1, double tot,
                                           double V, double h, int sub) {
  double v = tot > 0 ? V * p0.vol / tot : 0.5 * V;
  if (v > vmax0) v = vmax0;
  if (V - v > vmax1) v = V - vmax1;
  if (sub == 0) {
    S.vol[n0] = v;
    S.vol[n1] = V - v;
    store_solved(S, n0, h, p0.dv, p0);
    store_solved(S, n1, h, p1.dv, p1);
  }
}

// The level solve of the listed groups (levels.hpp:13-194). Groups are independent (a group's solve reads and writes only
// its members), so the team's level lane groups (32 / kLevelLanes<MIXED, W> per warp) take them as they come: each starts
// with the list entry of its own index, then takes the next one from the team's counter (S.misc[kMiscTaken]); groups
// take different numbers of passes, and a node's results do not depend on which lane group computes them. In 16-warp teams
// the upper warps, which have no buoyancy tree, start with the first entries.
//
// A unit needs its world extent to see that its starting level lies inside, and as the ends of the Newton bracket. Both are
// comparisons, which the first points of the extent lists mostly decide: a level above one of the bottoms is above the
// lowest, an iterate below one of the tops is below the highest. The rest of the lists are scanned only when they leave
// the question open or a bisection needs the ends themselves (and with a tape, which records the extent). A lane group's
// solver is a small machine (Phase) around one place for each of its parts.
template <bool MIXED, int W, class Tape>
__device__ __forceinline__ void solve_levels(const DevModel& M, const Pose& F, Slot& S, const Team<W>& T, const Tape& tape) {
  constexpr int LANES = kLevelLanes<MIXED, W>, PER_WARP = 32 / LANES;
  enum Phase { kIdle, kStart, kUpdate, kPass };
  const LevelLanes L = level_lanes<MIXED, W>(T.lane);
  const int grp = T.lane / LANES;
  PassR* const P = S.passes + static_cast<std::size_t>(T.warp * PER_WARP + grp) * M.maxGroup;
  const int listed = S.misc[kMiscListed];
  int i = (W == 16 ? T.warp ^ 8 : T.warp) * PER_WARP + grp;   // the next list entry
  int g0 = 0, g1 = 0;                          // the current group's first two members,
  const int* m = nullptr;                      // all of them when there are more than two,
  int N = 0, j = 0, units = 0;                 // their number, its next unit and its units
  bool merged = false;
  // the current unit: nm members, n0 and n1 first (the others from m) with their segments
  int n0 = 0, n1 = 0, nm = 0;
  int2 seg0{}, seg1{};
  // (phase is made opaque between the parts, or the compiler copies them for each phase they can follow: 3% of a full
  // load's time in code)
  // where its solve is: the member of the pass, the pass's tape slot, the Newton update, what is known of the extent
  int phase = kIdle;
  int k = 0, slot = 0, it = 0;
  bool full = false, empty = false, inside = false;
  bool aKnown = false, bKnown = false;  // a (b) is an iterate or the unit's whole extent's end, not just a first look's
  double V = 0, Vmax = 0, vmax1 = 0, h = 0, a = 0, b = 0, sum = 0, dvs = 0;
  auto member = [&](int q) { return q == 0 ? n0 : (q == 1 ? n1 : __ldg(m + q)); };
#pragma unroll 1
  for (;;) {
#pragma unroll 1
    while (phase == kIdle && (j < units || i < listed)) {
      if (j >= units) {
        g0 = g1 = S.list[i];
        int next = 0;
        if (L.sub == 0) next = atomicAdd(&S.misc[kMiscTaken], 1);
        i = __shfl_sync(L.mask, next, grp * LANES);
        N = 1;
        m = nullptr;
        merged = false;
        if (g0 >= kListedGroup) {
          const int g = g0 - kListedGroup;
          const uint2 bits = __ldg(reinterpret_cast<const uint2*>(M.groupEntry) + g);
          g0 = bits.x & 0xffff;
          g1 = bits.x >> 16;
          N = bits.y & 0xff;
          const int mode = (bits.y >> 8) & 0xff;
          if (N > 2) {
            if (N == 255) N = __ldg(M.gCount + g);
            m = M.gNodes + __ldg(M.gStart + g);
          }
          if (mode == 1) {
            merged = true;
          } else if (mode == 2) {
            const double zMw = world_z(F, __ldg(M.gpx + g), __ldg(M.gpy + g), __ldg(M.gpz + g));
            merged = true;
#pragma unroll 1
            for (int q = 0; q < N; ++q) {
              const int n = q == 0 ? g0 : (q == 1 ? g1 : __ldg(m + q));
              if (!(S.vol[n] > kEmptyVolume && group_level<MIXED, W>(M, S, n, L) > zMw + M.gMargin)) { merged = false; break; }
            }
          }
          if (L.sub == 0) S.merged[g] = merged ? 1 : 0;
        }
        units = merged ? 1 : N;
        j = 0;
      }
      n0 = j == 0 ? g0 : (j == 1 ? g1 : __ldg(m + j));
      nm = merged ? N : 1;
      n1 = nm > 1 ? g1 : n0;
      ++j;
      // everything the unit needs of its nodes' table, in one round of loads
      seg0 = __ldg(M.nodeSeg + n0); seg1 = __ldg(M.nodeSeg + n1);
      Vmax = __ldg(M.vmax + n0);
      V = S.vol[n0];
      vmax1 = __ldg(M.vmax + n1);
      if (nm > 1) { V += S.vol[n1]; Vmax += vmax1; }
#pragma unroll 1
      for (int q = 2; q < nm; ++q) { const int n = __ldg(m + q); V += S.vol[n]; Vmax += __ldg(M.vmax + n); }
      empty = V <= kEmptyVolume;
      if constexpr (Tape::kLazy) {
        if (empty) {
          if (L.sub == 0)
#pragma unroll 1
            for (int q = 0; q < nm; ++q) { const int n = member(q); S.dry[n] = (S.dry[n] & kStale) | kEmptyNode | (merged ? kZeroVolume : 0); }
          continue;
        }
      }
      // the starting level: the node's, the mean of a wet group's, or that of the group's first wet member (its last one
      // when none is)
      bool allWet = true;
      int firstWet = -1;
#pragma unroll 1
      for (int q = 0; merged && q < nm; ++q) {
        if (S.vol[member(q)] > 0) { if (firstWet < 0) firstWet = q; }
        else allWet = false;
      }
      const int q0 = allWet ? 0 : (firstWet >= 0 ? firstWet : nm - 1), q1 = allWet ? nm : q0 + 1;
      h = 0;
#pragma unroll 1
      for (int q = q0; q < q1; ++q) h += group_level<MIXED, W>(M, S, member(q), L);
      if (merged && allWet) h = nm == 2 ? 0.5 * h : h / static_cast<double>(nm);
      full = V >= Vmax * kFullFraction;
      inside = aKnown = bKnown = false;
      if (nm <= 2) {
        const Extents x = first_extents<MIXED, W>(M, F, n0, n1, nm == 2, L);
        a = nm == 2 && x.z[2] < x.z[0] ? x.z[2] : x.z[0];
        b = nm == 2 && x.z[3] > x.z[1] ? x.z[3] : x.z[1];
        inside = Tape::kLazy && !full && h >= a && h <= b;
        aKnown = bKnown = x.whole;
        if (inside || x.whole) {
          tape.start(n0, h, x.z[0], x.z[1], L);
          if (nm == 2) tape.start(n1, h, x.z[2], x.z[3], L);
          if (L.sub == 0) {
            const int flags = !Tape::kLazy && empty ? kEmptyNode | (merged ? kZeroVolume : 0) : kSolved | (x.whole ? 0 : kNoTop);
            S.zmax[n0] = x.z[1];
            S.dry[n0] = flags;
            if (nm == 2) { S.zmax[n1] = x.z[3]; S.dry[n1] = flags; }
            if (!Tape::kLazy && empty) { S.level[n0] = x.z[0]; if (nm == 2) S.level[n1] = x.z[2]; }
          }
        }
      }
      phase = kStart;
      break;
    }
    asm volatile("" : "+r"(phase));
    // an update's Newton iterate: sum and dvs are the unit's passes at h, the it-th after the starting one
    double hn = 0;
    if (phase == kUpdate) {
      const double err = sum - V;
      if (err > 0) { b = h; bKnown = true; } else { a = h; aKnown = true; }
      hn = h - err / dvs;
    }
    asm volatile("" : "+r"(phase));
    // the whole extent, where the first look leaves the start or an update open
    if ((phase == kStart && !inside && !aKnown) || (phase == kUpdate && !(aKnown && bKnown) && !(dvs > kSlopeMin && hn > a && hn < b))) {
      double lo = 0, hi = 0;
#pragma unroll 1
      for (int q = 0; q < nm; ++q) {
        const int n = member(q);
        double zlo = 0, zhi = 0;
#pragma unroll 1
        for (int top = 0; top < 2; ++top) {
          const double z = group_extreme<MIXED, W>(M, F, n, top != 0, L);
          if (top) zhi = z; else zlo = z;
        }
        if (q == 0 || zlo < lo) lo = zlo;
        if (q == 0 || zhi > hi) hi = zhi;
        if (phase == kStart) tape.start(n, h, zlo, zhi, L);
        if (L.sub == 0) {
          S.zmax[n] = zhi;
          S.dry[n] = !Tape::kLazy && empty ? kEmptyNode | (merged ? kZeroVolume : 0) : kSolved;
          if (!Tape::kLazy && empty) S.level[n] = zlo;
        }
      }
      if (!aKnown) a = lo;
      if (!bKnown) b = hi;
      aKnown = bKnown = true;
    }
    asm volatile("" : "+r"(phase));
    if (phase == kStart) {
      it = 0; slot = 0; k = 0; sum = 0; dvs = 0;
      phase = kPass;
      if (!Tape::kLazy && empty) {
        phase = kIdle;
      } else if (full) {
        // the pass at the top of a full unit, for its centroids; its level and volumes first
        double dh = 0;
        if (!merged) {
          dh = jmax(0.0, V - Vmax) / __ldg(M.aov + n0);
        } else {
          const double over = jmax(0.0, V - Vmax);
          double aSum = 0;
#pragma unroll 1
          for (int q = 0; q < nm; ++q) aSum += __ldg(M.aov + member(q));
          dh = over / aSum;
          if (L.sub == 0) {
            double assigned = 0;
#pragma unroll 1
            for (int q = 0; q < nm - 1; ++q) {
              const int n = member(q);
              const double v = __ldg(M.vmax + n) + dh * __ldg(M.aov + n);
              S.vol[n] = v;
              assigned += v;
            }
            S.vol[member(nm - 1)] = V - assigned;
          }
        }
        h = b;
        a = b + dh;  // the level
        slot = 1;
      } else if (!inside && (merged ? !(h >= a && h <= b) : (h < a || h > b))) {
        h = jmin(b, jmax(a, h));
        slot = 1;
      }
    } else if (phase == kUpdate) {
      if (!(dvs > kSlopeMin && hn > a && hn < b)) hn = 0.5 * (a + b);
      h = hn;
      ++it;
      sum = 0; dvs = 0;
      phase = kPass;
    }
    asm volatile("" : "+r"(phase));
    if (!__any_sync(kFull, phase == kPass)) {
      if (!__any_sync(kFull, j < units || i < listed)) break;
      continue;
    }
    int2 sg = k == 0 ? seg0 : seg1;
    int n = k == 0 ? n0 : n1;
    if (k > 1) { n = __ldg(m + k); sg = __ldg(M.nodeSeg + n); }
    if (phase != kPass) sg = int2{0, 0};
    const PassR p = node_pass<MIXED, W>(M, F, sg.x, sg.x + sg.y, __ldg(M.mu + n), h, L);
    if (phase != kPass) continue;
    tape.pass(n, slot, h, p, L);
    if (full) {
      if (L.sub == 0) store_solved(S, n, a, __ldg(M.aov + n), p);
      if (++k == nm) { phase = kIdle; k = 0; }
      continue;
    }
    sum += p.vol;
    dvs += p.dv;
    if (nm > 1) {
      if (L.sub == 0) P[k] = p;
      if (++k < nm) continue;
      k = 0;
    }
    ++slot;
    if (it < kNewtonFast && !(fabs(sum - V) < jmax(1e-3 * Vmax, 0.5))) {
      phase = kUpdate;
      continue;
    }
    if (nm == 2) {
      __syncwarp(L.mask);
      share_pair(S, P[0], p, n0, n1, __ldg(M.vmax + n0), vmax1, sum, V, h, L.sub);
    } else if (L.sub == 0) {
      if (nm == 1) store_solved(S, n, h, p.dv, p);
      else share_group(M, S, P, m, nm, V, h);
    }
    phase = kIdle;
  }
  __syncwarp();
}

// ----------------------------------------------------------------------------- flows (kernel/flows.hpp:38-78)
// Of a hull's connections most join two dry spaces or stand above the water (about 230 of titanic64's 290 early in a
// run), and a warp of 32 mixed ones issues the orifice's, the weir's and the submerged weir's code (two pow) one after
// the other. Teams of up to four warps, of which many share an SM and issue slots bound it, therefore sort them first
// (sort_connections): the ones that can flow go into a list whose front holds orifices and free weirs and whose back
// holds submerged weirs, the others' flow is zero; then the listed ones are computed, a warp's lanes in one class.
// Larger teams have a thread for every connection of such a hull and are bound by the chain of dependent steps: they
// form every flow while they count the degrees, and limit it after the barrier (team_step). A node's reciprocal area is
// divided once, and a monitor divides the flows it sums itself (the step kept every connection's quotient before).
// On B200, when it came: 2,048 uneven titanic64 runs to 20 min 469 ms against 493 (two-warp teams); one run to 5 min 32.2
// against 33.4 (the sorted form in its 16-warp team: 35.4), 264 liner runs to 15 min 113 against 114 (sorted: 123). With the
// present step the two forms are level in between: 4 warps, 500 titanic64 runs to 5 min 38.3 sorted, 38.2 not; 8 warps, 250
// runs to 1 min 4.13 sorted, 4.11 not.

// The heads over connection c's opening at its two ends.
struct FlowHeads {
  int a, b;
  double zo, Ha, Hb;
};

__device__ __forceinline__ FlowHeads flow_heads(const DevModel& M, const Pose& F, const Slot& S, int c) {
  FlowHeads f;
  f.a = __ldg(M.ca + c);
  f.b = __ldg(M.cb + c);
  f.zo = F.R20 * __ldg(M.kx + c) + F.R21 * __ldg(M.ky + c) + F.R22 * __ldg(M.kz + c) + F.tz;
  const double ha = f.a < 0 ? 0.0 : S.hEff[f.a], hb = S.hEff[f.b];
  f.Ha = ha > f.zo ? ha - f.zo : 0.0;
  f.Hb = hb > f.zo ? hb - f.zo : 0.0;
  return f;
}

// Node n's degree, in the first half of its place in S.acc (zeroed with the heads, dead with the volume update).
__device__ __forceinline__ int* degree(const Slot& S, int n) { return reinterpret_cast<int*>(S.acc + n); }

// A node's degree is the number of its incident connections that are enabled and not between two empty spaces. Each such
// connection counts once at each of its nodes (the incidence lists hold it once at a when a >= 0 and once at b), counted
// per connection with shared-memory atomics: an integer count, the same in any order, and one round of independent loads
// instead of a walk down every node's incidence list. Returns whether connection c may flow at time t (an uncounted one
// cannot: both its ends are empty).
template <class IP>
__device__ __forceinline__ bool count_degrees(const DevModel& M, double t, Slot& S, const IP& I, int c) {
  if (!__ldg(I.en() + c)) return false;
  const int a = __ldg(M.ca + c), b = __ldg(M.cb + c);
  if (a >= 0 && S.hEff[a] < kNoHeadTest && S.hEff[b] < kNoHeadTest) return false;
  if (a >= 0) atomicAdd(degree(S, a), 1);
  atomicAdd(degree(S, b), 1);
  const int sk = __ldg(M.skip + c);
  return !(__ldg(I.tOn() + c) > t) && !(sk >= 0 && S.merged[sk]);
}

// The volume that connection c's law sends through it in the step, a to b.
__device__ __forceinline__ double law_volume(const DevModel& M, const FlowHeads& f, const double* area, int c) {
  const double Ha = f.Ha, Hb = f.Hb;
  double q = 0;
  if (__ldg(M.law + c) == 0) {
    const double d = Ha - Hb;
    if (d != 0) q = __ldg(M.coef + c) * __ldg(area + c) * M.sq2g * d / pm::sqrt_rn(jmax(fabs(d), kOrificeHeadFloor));
  } else {
    const double H1 = Ha > Hb ? Ha : Hb;
    if (H1 > 0) {
      const double H2 = Ha > Hb ? Hb : Ha;
      double v = 1;
      if (H2 > 0) {
        const double r = H2 / H1;
        v = pow_of(jmax(0.0, 1 - pow_of(r, kWeirExponent)), kVillemonteExponent);
      }
      q = __ldg(M.coef + c) * __ldg(area + c) * kWeirCoefficient * M.sq2g * H1 * pm::sqrt_rn(H1) * v * (Ha >= Hb ? 1.0 : -1.0);
    }
  }
  return q == 0 ? 0 : q * M.dt;
}

// The flow dV (not zero) after the limiter. S.aEff holds the reciprocals of the nodes' effective areas.
__device__ __forceinline__ double limit_volume(const Slot& S, const FlowHeads& f, double dV) {
  const int src = dV > 0 ? f.a : f.b, dst = dV > 0 ? f.b : f.a;
  const double hs = src < 0 ? 0.0 : S.hEff[src];
  const double hd = dst < 0 ? 0.0 : S.hEff[dst];
  const double inv = (src < 0 ? 0.0 : S.aEff[src]) + (dst < 0 ? 0.0 : S.aEff[dst]);
  const int degSrc = src < 0 ? 0 : *degree(S, src), degDst = dst < 0 ? 0 : *degree(S, dst);
  const int degRef = degSrc > degDst ? degSrc : degDst;
  const double share = kLimiterShare / static_cast<double>(degRef > 1 ? degRef : 1);
  double lim = inv > 0 ? share * (hs - jmax(hd, f.zo)) / inv : fabs(dV);
  if (lim < 0) lim = 0;
  if (fabs(dV) > lim) dV = dV > 0 ? lim : -lim;
  return dV;
}

// Sorts the connections (zero, front or back) and counts the nodes' degrees; the flows follow after a barrier
// (listed_flows). The order within the list varies, the flows do not depend on it.
template <int W, class IP>
__device__ __forceinline__ void sort_connections(const DevModel& M, const Pose& F, double t, Slot& S, const IP& I, const Team<W>& T) {
#pragma unroll 1
  for (int c0 = T.warp * kLanes; c0 < M.nc; c0 += kLanes * W) {
    const int c = c0 + T.lane;
    int cls = 0;
    if (c < M.nc) {
      S.dV[c] = 0;
      if (count_degrees(M, t, S, I, c)) {
        const FlowHeads f = flow_heads(M, F, S, c);
        if (__ldg(M.law + c) == 0) {
          cls = f.Ha - f.Hb != 0 ? 1 : 0;
        } else if ((f.Ha > f.Hb ? f.Ha : f.Hb) > 0) {
          cls = (f.Ha > f.Hb ? f.Hb : f.Ha) > 0 ? 2 : 1;
        }
      }
    }
    const unsigned front = __ballot_sync(kFull, cls == 1), back = __ballot_sync(kFull, cls == 2);
    const unsigned before = (1u << T.lane) - 1u;
    if (front) {
      int base = 0;
      if (T.lane == 0) base = atomicAdd(&S.misc[kMiscFront], __popc(front));
      base = __shfl_sync(kFull, base, 0);
      if (cls == 1) S.flow[base + __popc(front & before)] = static_cast<std::uint16_t>(c);
    }
    if (back) {
      int base = 0;
      if (T.lane == 0) base = atomicAdd(&S.misc[kMiscBack], __popc(back));
      base = __shfl_sync(kFull, base, 0);
      if (cls == 2) S.flow[M.nc - 1 - (base + __popc(back & before))] = static_cast<std::uint16_t>(c);
    }
  }
}

template <int W, class IP>
__device__ __forceinline__ void listed_flows(const DevModel& M, const Pose& F, Slot& S, const IP& I, const Team<W>& T) {
  const int front = S.misc[kMiscFront], back = S.misc[kMiscBack];
  const int split = (front + kLanes - 1) / kLanes * kLanes;  // the back starts with a new warp
#pragma unroll 1
  for (int k = T.rank; k < split + back; k += kLanes * W) {
    if (k >= front && k < split) continue;
    const int c = S.flow[k < front ? k : M.nc - 1 - (k - split)];
    const FlowHeads f = flow_heads(M, F, S, c);
    const double dV = law_volume(M, f, I.area(), c);
    S.dV[c] = dV != 0 ? limit_volume(S, f, dV) : dV;
  }
}

// Scalars of one simulation: identical in every lane of its warp.
struct SimRegs {
  double t, zO, pitch, roll, vz, wth, wph, calm;
  double inflow, Vb, hullTop, mw, bx, by, bz;
  int foundered;
  double founderT;
  int evCount;  // the event warp's count is the log's; the other warps' lag
};

// The run's values live in the slot (Parked) through a step, so that their registers serve its phases; the step's first
// warp moves them on, and every thread takes them at its end. The settle timer and the event count stay in registers.
__device__ __forceinline__ void park(Parked* P, const SimRegs& R) {
  P->t = R.t; P->zO = R.zO; P->pitch = R.pitch; P->roll = R.roll; P->vz = R.vz; P->wth = R.wth; P->wph = R.wph;
  P->inflow = R.inflow; P->Vb = R.Vb; P->hullTop = R.hullTop; P->mw = R.mw; P->bx = R.bx;
  P->by = R.by; P->bz = R.bz; P->founderT = R.founderT; P->foundered = R.foundered;
}

__device__ __forceinline__ void unpark(const Parked* P, SimRegs& R) {
  R.t = P->t; R.zO = P->zO; R.pitch = P->pitch; R.roll = P->roll; R.vz = P->vz; R.wth = P->wth; R.wph = P->wph;
  R.inflow = P->inflow; R.Vb = P->Vb; R.hullTop = P->hullTop; R.mw = P->mw; R.bx = P->bx;
  R.by = P->by; R.bz = P->bz; R.founderT = P->founderT; R.foundered = P->foundered;
}

// Instance `inst`'s per-instance arrays. In a batch of one model each pointer is formed where it is used from the
// batch's base pointers (kernel parameters) and inst x the model's sizes, so a thread holds one index rather than
// eight pointers through the step; in a fleet (FLEET) the instance's offsets are loaded once when it is claimed.
template <bool FLEET>
struct InstPtrs;

template <>
struct InstPtrs<false> {
  const DevModel& M;
  const DevBatch& B;
  int inst;
  __device__ __forceinline__ std::size_t perConn() const { return static_cast<std::size_t>(inst) * M.nc; }
  __device__ __forceinline__ std::size_t perEvent() const { return static_cast<std::size_t>(inst) * M.evCap; }
  __device__ __forceinline__ std::size_t perNode() const { return static_cast<std::size_t>(inst) * M.nn; }
  __device__ __forceinline__ std::size_t perMonitor() const { return static_cast<std::size_t>(inst) * M.nmon; }
  __device__ __forceinline__ std::size_t perMark() const { return static_cast<std::size_t>(inst) * M.nmark; }
  __device__ __forceinline__ const std::uint8_t* en() const { return B.en + perConn(); }
  __device__ __forceinline__ const double* area() const { return B.area + perConn(); }
  __device__ __forceinline__ const double* tOn() const { return B.tOn + perConn(); }
  __device__ __forceinline__ double* evT() const { return B.evT + perEvent(); }
  __device__ __forceinline__ std::int32_t* evId() const { return B.evId + perEvent(); }
  __device__ __forceinline__ std::int32_t* evKind() const { return B.evKind + perEvent(); }
  __device__ __forceinline__ double* overT() const { return B.overT + perMonitor(); }
  __device__ __forceinline__ double* markT() const { return B.markT + perMark(); }
};

template <>
struct InstPtrs<true> {
  const DevModel& M;
  const DevBatch& B;
  int inst;
  const std::uint8_t* en_;
  const double *area_, *tOn_;
  double *evT_, *overT_, *markT_;
  std::int32_t *evId_, *evKind_;
  std::size_t node_;
  __device__ __forceinline__ InstPtrs(const DevModel& m, const DevBatch& b, int i) : M(m), B(b), inst(i) {
    const std::size_t c = static_cast<std::size_t>(B.connOff[i]), e = static_cast<std::size_t>(B.evOff[i]);
    en_ = B.en + c; area_ = B.area + c; tOn_ = B.tOn + c;
    evT_ = B.evT + e; evId_ = B.evId + e; evKind_ = B.evKind + e;
    overT_ = B.overT + B.monOff[i]; markT_ = B.markT + B.markOff[i];
    node_ = static_cast<std::size_t>(B.nodeOff[i]);
  }
  __device__ __forceinline__ std::size_t perNode() const { return node_; }
  __device__ __forceinline__ const std::uint8_t* en() const { return en_; }
  __device__ __forceinline__ const double* area() const { return area_; }
  __device__ __forceinline__ const double* tOn() const { return tOn_; }
  __device__ __forceinline__ double* evT() const { return evT_; }
  __device__ __forceinline__ std::int32_t* evId() const { return evId_; }
  __device__ __forceinline__ std::int32_t* evKind() const { return evKind_; }
  __device__ __forceinline__ double* overT() const { return overT_; }
  __device__ __forceinline__ double* markT() const { return markT_; }
};

// The event log belongs to one warp of the team (not the first where there are two: that one integrates the motion
// meanwhile); its lane 0 writes, only its count is stored.
template <int W>
constexpr int kEventWarp = W > 1 ? 1 : 0;

template <class IP>
__device__ __forceinline__ void push_event(const DevModel& M, double t, int& evCount, const IP& I, int id, int kind, int lane) {
  if (evCount < M.evCap) {
    if (lane == 0) { I.evT()[evCount] = t; I.evId()[evCount] = id; I.evKind()[evCount] = kind; }
    evCount++;
  }
}

// The overflow and mark events of a step that ends at time t (events.hpp:11-38): monitors in order, then marks in order,
// at the step's pose and flows. One warp.
template <class IP>
__device__ __forceinline__ void step_events(const DevModel& M, const Pose& F, double t, int& evCount, const Slot& S, const IP& I, int lane) {
#pragma unroll 1
  for (int m0 = 0; m0 < M.nmon; m0 += kLanes) {
    const int m = m0 + lane;
    bool fire = false;
    if (m < M.nmon && I.overT()[m] < 0) {
      const int k0 = __ldg(M.monStart + m), k1 = k0 + __ldg(M.monCount + m);
      double over = 0;
#pragma unroll 1
      for (int k = k0; k < k1; ++k) {
        const double d = S.dV[__ldg(M.monConn + k)];
        if (d > 0) over += d / M.dt;
      }
      fire = over > M.monThreshold;
      if (fire) I.overT()[m] = t;
    }
    unsigned mask = __ballot_sync(kFull, fire);
    while (mask) {
      const int b = __ffs(mask) - 1;
      mask &= mask - 1;
      push_event(M, t, evCount, I, m0 + b, 0, lane);
    }
  }
#pragma unroll 1
  for (int i0 = 0; i0 < M.nmark; i0 += kLanes) {
    const int i = i0 + lane;
    bool fire = false;
    if (i < M.nmark && I.markT()[i] < 0) {
      const double wz = world_z(F, __ldg(M.mkx + i), __ldg(M.mky + i), __ldg(M.mkz + i));
      const bool under = __ldg(M.mkWhen + i) == 0;
      fire = (under && wz < 0) || (!under && wz > 0);
      if (fire) I.markT()[i] = t;
    }
    unsigned mask = __ballot_sync(kFull, fire);
    while (mask) {
      const int b = __ffs(mask) - 1;
      mask &= mask - 1;
      push_event(M, t, evCount, I, i0 + b, 1, lane);
    }
  }
}

// The sum of the nonzero values of v over the lanes, in lane order, added to (or, with SUB, taken from) acc; zeros leave
// a sum as it is.
template <bool SUB>
__device__ __forceinline__ double add_in_order(double acc, double v) {
  unsigned mask = __ballot_sync(kFull, v != 0);
  while (mask) {
    const int b = __ffs(mask) - 1;
    mask &= mask - 1;
    const double x = __shfl_sync(kFull, v, b);
    acc = SUB ? acc - x : acc + x;
  }
  return acc;
}

// ----------------------------------------------------------------------------- the step (kernel/step.hpp:41-54)
// Phases that exchange per-node or per-connection arrays are separated by team barriers; per-node and
// per-connection work is spread over all 32 W threads of the team; the sums over nodes in their serial order, the
// motion and the next pose are one warp's, while another lists the next solve's groups and a third the events.

// The inflow from the sea in the step that just flowed (flows.hpp:114-118): the sea connections in order, less the excess
// that returns, in node order. Nothing in the motion needs it, so another warp forms it meanwhile.
__device__ __forceinline__ void sea_inflow(const DevModel& M, Slot& S, int lane) {
  double seaIn = 0;
#pragma unroll 1
  for (int k0 = 0; k0 < M.nsea; k0 += kLanes) {
    const int k = k0 + lane;
    seaIn = add_in_order<false>(seaIn, k < M.nsea ? S.dV[__ldg(M.sea + k)] : 0.0);
  }
#pragma unroll 1
  for (int n0 = 0; n0 < M.nn; n0 += kLanes) {
    const int n = n0 + lane;
    seaIn = add_in_order<true>(seaIn, n < M.nn && S.acc[n] > 0 ? S.acc[n] : 0.0);
  }
  if (lane == 0) S.parked->inflow = seaIn / M.dt;
}

// The semi-implicit motion (body.hpp:42-57) and the founder rule (events.hpp:30-38) on the run's values, by the lanes of one
// warp alike; returns (zO, pitch, roll).
struct MotionIn {
  double tauX, tauY, Fz, mw, Iwp, Iwr, cth;
};

__device__ __forceinline__ double3 integrate_motion(const DevModel& M, Parked& P, const MotionIn& I, const Buoy& hb) {
  const double Mth = I.tauY, Mph = I.tauX * I.cth;
  const double dt = M.dt;
  double vz = P.vz, wth = P.wth, wph = P.wph, zO = P.zO, pitch = P.pitch, roll = P.roll;
  const double mh = M.mh0 + I.mw;
  const double Ith = M.Ith0 + I.Iwp, Iph = M.Iph0 + I.Iwr;
  const double az = (I.Fz - M.cDz * vz - M.qz * fabs(vz) * vz) / mh;
  const double ath = (Mth - M.cDth * wth - M.qth * fabs(wth) * wth) / Ith;
  const double aph = (Mph - M.cDph * wph - M.qph * fabs(wph) * wph) / Iph;
  vz += az * dt; wth += ath * dt; wph += aph * dt;
  zO += vz * dt; pitch += wth * dt; roll += wph * dt;
  if (pitch > kPitchClamp) { pitch = kPitchClamp; wth = 0; }
  if (pitch < -kPitchClamp) { pitch = -kPitchClamp; wth = 0; }
  if (roll > kRollClamp) { roll = kRollClamp; wph = 0; }
  if (roll < -kRollClamp) { roll = -kRollClamp; wph = 0; }
  const double t = P.t + dt;
  __syncwarp();  // the lanes have read the values they now replace
  P.t = t; P.zO = zO; P.pitch = pitch; P.roll = roll; P.vz = vz; P.wth = wth; P.wph = wph;
  P.Vb = hb.V; P.hullTop = hb.top; P.mw = I.mw;
  P.bx = hb.x; P.by = hb.y; P.bz = hb.z;
  if (!P.foundered && (hb.top < M.hullTopBelow || fabs(pitch) > M.pitchAbsAbove || (hb.V < M.buoyancyBelow && t > M.minT))) {
    P.foundered = 1;
    P.founderT = t;
  }
  return double3{zO, pitch, roll};
}

// The load sums, the motion and the next pose (body.hpp:11-57, events.hpp:30-38), by one warp. The load terms of the
// flooded nodes are in five columns a fixed stride apart from S.area, in node order, 32 nodes' at the front of their 32
// places and their number in S.wet (team_step). Lanes 0 .. 5 each add one column: a lane reading all of them, node by node,
// took a dependent load and six adds for each of all the nodes, and an add takes 23 cycles. The third column holds volumes,
// of which lane 2 adds the weights and lane 3 the masses; the others' factor of one leaves their terms as they are.
__device__ __forceinline__ void move_body(const DevModel& M, const Pose& F, Slot& S, int lane) {
  Parked& P = *S.parked;
  const Buoy hb = buoyancy_finish(S.hydro);
  const double Wg = M.rho * M.g;
  const double Fb = Wg * hb.V;
  const double bxw = F.R00 * hb.x + F.R01 * hb.y + F.R02 * hb.z + F.tx;
  const double byw = F.R10 * hb.x + F.R11 * hb.y + F.R12 * hb.z + F.ty;
  double sum = 0;
  if (lane == 0) sum = (byw - M.YO) * Fb;
  if (lane == 1) sum = -(bxw - M.XO) * Fb;
  if (lane == 2) sum = Fb - M.g * M.ms;
  {
    // (min, not nested choices: those cost the 16-warp fleet kernel 248 bytes of spills, 96 ships to 5 min 32 ms against 24.4)
    const double* t = S.area + min(lane - (lane >= 3 ? 1 : 0), 4) * (S.zmax - S.area);
    const double factor = lane == 2 ? -Wg : (lane == 3 ? M.rho : 1.0);
#pragma unroll 1
    for (int n0 = 0; n0 < M.nn; n0 += kLanes) {
      const int wet = S.wet[n0 / kLanes];
#pragma unroll 4
      for (int k = 0; k < wet; ++k) sum += factor * t[n0 + k];
    }
  }
  const double tauX = __shfl_sync(kFull, sum, 0), tauY = __shfl_sync(kFull, sum, 1), Fz = __shfl_sync(kFull, sum, 2);
  const double mw = __shfl_sync(kFull, sum, 3), Iw_p = __shfl_sync(kFull, sum, 4), Iw_r = __shfl_sync(kFull, sum, 5);
  const MotionIn in{tauX, tauY, Fz, mw, Iw_p, Iw_r, F.cth};
  const double3 at = integrate_motion(M, P, in, hb);
  *S.prev = make_pose(M, at.x, at.y, at.z);
}

// One step. On entry S.parked holds R's values and S.pose their pose; on return R, S.parked and S.pose are the next ones
// (S.prev the step's).
template <bool MIXED, int W, class IP, class Tape = NoTape>
__device__ __forceinline__ void team_step(const DevModel& M, SimRegs& R, Slot& S, const IP& I, const Team<W>& T, const Tape& tape = Tape{}) {
  constexpr int kStride = 32 * W;
  const int lane = T.lane, rank = T.rank;
  const Pose& F = *S.pose;
  buoyancy_trees<MIXED, W>(M, F, T.warp, lane, S.hydro, S.cols);
  // The buoyancy's eight trees and the level solve need nothing from each other: in 16-warp teams the warps without a
  // tree go on to take list entries, and one barrier ends both. In smaller teams every warp has trees, and a barrier
  // between keeps the warps in the same tables.
  if constexpr (W <= 8) T.sync();
  solve_levels<MIXED, W>(M, F, S, T, tape);
  T.sync();
  // the list counter for the next step's level solve (read after this step's later barriers)
  if (T.leader()) {
    S.misc[kMiscTaken] = W * (32 / kLevelLanes<MIXED, W>);
    S.misc[kMiscFront] = 0;
    S.misc[kMiscBack] = 0;
  }

  // the solve's ends node by node (an empty node's area, a wet one's centroid), effective heads and areas, then degrees
  // (flows.hpp:15-35)
#pragma unroll 1
  for (int n = rank; n < M.nn; n += kStride) {
    const int flags = S.dry[n];
    S.dry[n] = Tape::kLazy ? ((flags & kEmptyNode) ? kStale : flags & kNoTop) : 0;
    if (flags & kEmptyNode) {
      S.area[n] = 0;
      if (flags & kZeroVolume) S.vol[n] = 0;
    } else if (flags & kSolved) {
      set_centroid(S, n);
    }
    const double v = S.vol[n];
    S.hEff[n] = v > kEmptyVolume ? S.level[n] : kNoHead;
    S.aEff[n] = 1 / (v >= __ldg(M.vmax + n) ? __ldg(M.aov + n) : jmax(S.area[n], __ldg(M.amin + n)));
    S.acc[n] = 0;  // the degree
  }
  tape.solved(M, S, T);  // a thread reads the nodes it has just finished
  T.sync();
  const double tNow = S.parked->t;
  if constexpr (W <= 4) {
    sort_connections(M, F, tNow, S, I, T);
    T.sync();
    listed_flows(M, F, S, I, T);
  } else {
#pragma unroll 1
    for (int c = rank; c < M.nc; c += kStride)
      S.dV[c] = count_degrees(M, tNow, S, I, c) ? law_volume(M, flow_heads(M, F, S, c), I.area(), c) : 0;
    T.sync();
#pragma unroll 1
    for (int c = rank; c < M.nc; c += kStride) {
      const double dV = S.dV[c];
      if (dV != 0) S.dV[c] = limit_volume(S, flow_heads(M, F, S, c), dV);
    }
  }
  T.sync();
  // per-node gathers in increasing connection order, the volume update (flows.hpp:81-111) and, by the same thread, the
  // node's terms of the loads (body.hpp:20-33), which overwrite arrays of which only these 32 nodes' entries are still read
  // (and those before the ballot)
  {
    const double Wg = M.rho * M.g;
    const double zO = S.parked->zO;
#pragma unroll 1
    for (int n0 = T.warp * kLanes; n0 < M.nn; n0 += kStride) {
      const int n = n0 + lane < M.nn ? n0 + lane : n0;
      const int k0 = __ldg(M.incStart + n), k1 = n0 + lane < M.nn ? k0 + __ldg(M.incCount + n) : k0;
      double acc = 0;
#pragma unroll 4
      for (int k = k0; k < k1; ++k) {
        const int e = __ldg(M.incEdge + k);
        const double d = S.dV[e >> 1];
        acc = (e & 1) ? acc + d : acc - d;
      }
      double v = S.vol[n] + acc;
      if (v < 0) v = 0;
      const double vm = __ldg(M.vmax + n);
      double excess = 0;
      if (v > vm) {
        // (a node that was empty at the solve, or whose solve did not need it, has no highest point yet)
        const double zmax = (S.dry[n] & (kStale | kNoTop)) ? static_cast<double>(node_extreme<MIXED>(M, F, n, true, 0, 1)) : S.zmax[n];
        const double head = jmax(0.0, -zmax);
        const double cap = vm + __ldg(M.aov + n) * head;
        if (v > cap) { excess = v - cap; v = cap; }
      }
      const bool mine = n0 + lane < M.nn, wet = mine && !(v <= 0);
      const unsigned mask = __ballot_sync(kFull, wet);
      if (lane == 0) S.wet[n0 / kLanes] = static_cast<std::uint8_t>(__popc(mask));
      if (mine) {
        S.acc[n] = excess;
        S.vol[n] = v;
      }
      if (wet) {
        const double x = S.cx[n], y = S.cy[n], z = S.cz[n];
        const double wx = F.R00 * x + F.R01 * y + F.R02 * z + F.tx - M.XO;
        const double wy = F.R10 * x + F.R11 * y + F.R12 * z + F.ty - M.YO;
        const double wz = F.R20 * x + F.R21 * y + F.R22 * z + F.tz - zO;
        const double f = -Wg * v;
        const double m = M.rho * v;
        const int at = n0 + __popc(mask & ((1u << lane) - 1u));
        S.area[at] = wy * f;
        S.zmax[at] = -(wx * f);
        S.hEff[at] = v;
        S.aEff[at] = m * (wx * wx + wz * wz);
        S.tmp[at] = m * (wy * wy + wz * wz);
      }
    }
  }
  T.sync();
  if (T.warp == 0) move_body(M, F, S, lane);
  if constexpr (Tape::kLazy) {
    if (T.warp == W - 1) list_groups<true>(M, S, lane);
  }
  if (T.warp == kEventWarp<W>) step_events(M, F, tNow + M.dt, R.evCount, S, I, lane);
  if (T.warp == (W > 2 ? 2 : W - 1)) sea_inflow(M, S, lane);
  T.sync();
  Pose* const last = S.pose;
  S.pose = S.prev;
  S.prev = last;
  unpark(S.parked, R);
  if (R.foundered && T.warp == kEventWarp<W>) push_event(M, R.t, R.evCount, I, -1, 2, lane);
}

// Readouts at the current state (kernel/readouts.hpp:20-36): t, trim, list, water (t), inflow (t/min), draftF, draftA.
__device__ __forceinline__ void readouts(const DevModel& M, const SimRegs& R, const Slot& S, double* r7) {
  const Pose F = make_pose(M, R.zO, R.pitch, R.roll);
  double water = 0;
#pragma unroll 1
  for (int n = 0; n < M.nn; ++n) water += S.vol[n];
  r7[0] = R.t;
  r7[1] = R.pitch * 180 / kPi;
  r7[2] = R.roll * 180 / kPi;
  r7[3] = water * M.rho / 1000;
  r7[4] = R.inflow * M.rho / 1000 * 60;
  r7[5] = -world_z(F, M.xFP, 0, 0);
  r7[6] = -world_z(F, M.xAP, 0, 0);
}

}  // namespace ssb
