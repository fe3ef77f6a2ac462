// Device memory of one compiled model and of the buffers the engines own: DevBuf (an owning device array) and ModelDev
// (a compiled ship and sim in the kernels' layout, DevModel pointing into it). Shared by the batch engine (batch.cpp)
// and the adjoint engine (adjoint.cpp).
#pragma once

#include <algorithm>
#include <cmath>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "device_model.h"
#include "extents.h"
#include "model.h"

namespace ssb {

inline void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA: ") + what + ": " + cudaGetErrorString(e));
}


// A device array that owns its allocation.
template <class T>
class DevBuf {
 public:
  DevBuf() = default;
  ~DevBuf() { release(); }
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  void alloc(std::size_t n) {
    if (p_ && n == n_) return;  // same size: keep the allocation (a re-run reuses every buffer)
    release();
    n_ = n;
    if (n) check(cudaMalloc(reinterpret_cast<void**>(&p_), n * sizeof(T)), "cudaMalloc");
  }
  void upload(const std::vector<T>& v, cudaStream_t s) {
    if (v.size() != n_) alloc(v.size());
    if (n_) check(cudaMemcpyAsync(p_, v.data(), n_ * sizeof(T), cudaMemcpyHostToDevice, s), "copy to device");
  }
  void download(std::vector<T>& v, cudaStream_t s) const {
    v.resize(n_);
    if (n_) check(cudaMemcpyAsync(v.data(), p_, n_ * sizeof(T), cudaMemcpyDeviceToHost, s), "copy to host");
  }
  T* get() const { return p_; }
  std::size_t size() const { return n_; }
  std::size_t bytes() const { return n_ * sizeof(T); }

 private:
  T* p_ = nullptr;
  std::size_t n_ = 0;
  void release() {
    if (p_) cudaFree(p_);
    p_ = nullptr;
    n_ = 0;
  }
};


inline std::uint32_t take(std::uint32_t& off, std::size_t bytes) {
  const std::uint32_t at = off;
  off = static_cast<std::uint32_t>((off + bytes + 15) & ~static_cast<std::size_t>(15));
  return at;
}

// The shared-memory slot of one simulation of a model of these sizes, stepped by a team of W warps: per-node state and
// scratch, the connections' flows and their list, the group-pass buffers, the buoyancy tree results, the poses and
// parked run values, and in a fleet the team's copy of its instance's model.
inline SlotLayout slot_layout(std::int32_t NN, std::int32_t NC, std::int32_t NG, std::int32_t maxGroup, int W, bool fleet) {
  SlotLayout L{};
  std::uint32_t off = 0;
  const std::size_t nb = sizeof(double) * static_cast<std::size_t>(NN);
  const std::size_t cb = sizeof(double) * static_cast<std::size_t>(std::max(NC, 1));
  L.vol = take(off, nb); L.level = take(off, nb); L.cx = take(off, nb); L.cy = take(off, nb); L.cz = take(off, nb);
  // six columns that the loads' terms are summed down side by side, so a stride that puts them in different banks
  const std::size_t column = sizeof(double) * ((static_cast<std::size_t>(NN) + 5) / 8 * 8 + 2);
  L.area = take(off, column); L.zmax = take(off, column); L.hEff = take(off, column); L.aEff = take(off, column); L.tmp = take(off, column);
  L.term5 = take(off, column);
  L.acc = take(off, nb);
  L.deg = take(off, sizeof(std::int32_t) * static_cast<std::size_t>(NN));
  L.dV = take(off, cb);
  L.flow = take(off, sizeof(std::uint16_t) * static_cast<std::size_t>(std::max(NC, 1)));
  L.passes = take(off, 5 * sizeof(double) * static_cast<std::size_t>(maxGroup) * static_cast<std::size_t>(W * kMaxLevelGroupsPerWarp));
  L.hydro = take(off, 33 * sizeof(double));
  L.misc = take(off, 8 * sizeof(std::int32_t));
  L.merged = take(off, static_cast<std::size_t>(std::max(NG, 1)));
  L.dry = take(off, static_cast<std::size_t>(std::max(NN, 1)));
  L.wet = take(off, static_cast<std::size_t>(NN) / 32 + 1);
  L.list = take(off, sizeof(Listed) * static_cast<std::size_t>(std::max(NG, 1)));
  L.pose = take(off, 2 * sizeof(Pose));
  L.parked = take(off, sizeof(Parked));
  L.model = fleet ? take(off, sizeof(DevModel)) : 0u;
  L.bytes = off;
  return L;
}

// One compiled model on the device: its geometry in the kernel's layout (paired fields, the segment -> column gather
// resolved, float copies), its node, group, connection, incidence, monitor and mark tables, and the DevModel that
// points into them.
struct ModelDev {
  std::shared_ptr<const CompiledShip> ship;
  CompiledSim sim;
  Incidence inc;
  MonitorLists mons;
  std::int32_t NN = 0, NC = 0, NG = 0, nmon = 0, nmark = 0, evCap = 0, maxGroup = 0;
  DevBuf<double2> colXY, colLH, segXY, segLH, exXY;
  DevBuf<float2> colXYf, colLHf, segXYf, segLHf, exXYf;
  DevBuf<float> colAf, segArf, exZf;
  DevBuf<double> colA, segAr, exZ, mu, vmax, amin, aov;
  DevBuf<std::int32_t> exStart, incEdge, segStart, segCount, gStart, gCount, gNodes, ca, cb, skip, incStart, incCount, incConn, sea, monStart, monCount, monConn;
  DevBuf<int2> nodeSeg;
  DevBuf<Listed> groupEntry;
  DevBuf<std::uint8_t> gMode, law, incSide, mkWhen;
  DevBuf<double> gpx, gpy, gpz, kx, ky, kz, coef, mkx, mky, mkz;
  DevModel dm{};

  ModelDev(std::shared_ptr<const CompiledShip> s, const CompiledSim& m) : ship(std::move(s)), sim(m) {
    if (!ship) throw std::invalid_argument("Batch: null ship");
    check_pairing(*ship, sim);
    inc = build_incidence(sim);
    mons = build_monitor_lists(sim);
    NN = ship->nodes(); NC = sim.connections(); NG = sim.groups();
    nmon = sim.monitors(); nmark = sim.marks(); evCap = nmon + nmark + 1; maxGroup = sim.maxGroupSize();
  }

  void upload(cudaStream_t s) {
    const CompiledShip& S = *ship;
    const CompiledSim& M = sim;
    {
      const std::size_t nc = S.x.size(), ns = S.segCol.size();
      std::vector<double2> cxy(nc), clh(nc), sxy(ns), slh(ns);
      std::vector<float2> cxyf(nc), clhf(nc), sxyf(ns), slhf(ns);
      std::vector<double> sa(ns);
      std::vector<float> caf(nc), saf(ns);
      for (std::size_t i = 0; i < nc; ++i) {
        cxy[i] = double2{S.x[i], S.y[i]};
        clh[i] = double2{S.zlo[i], S.zhi[i]};
        cxyf[i] = float2{static_cast<float>(S.x[i]), static_cast<float>(S.y[i])};
        clhf[i] = float2{static_cast<float>(S.zlo[i]), static_cast<float>(S.zhi[i])};
        caf[i] = static_cast<float>(S.dxdy[i]);
      }
      for (std::size_t j = 0; j < ns; ++j) {
        const auto c = static_cast<std::size_t>(S.segCol[j]);
        sxy[j] = double2{S.x[c], S.y[c]};
        slh[j] = double2{S.segA[j], S.segE[j]};
        sa[j] = S.dxdy[c];
        sxyf[j] = float2{static_cast<float>(S.x[c]), static_cast<float>(S.y[c])};
        slhf[j] = float2{static_cast<float>(S.segA[j]), static_cast<float>(S.segE[j])};
        saf[j] = static_cast<float>(S.dxdy[c]);
      }
      colXY.upload(cxy, s); colLH.upload(clh, s); colA.upload(S.dxdy, s);
      colXYf.upload(cxyf, s); colLHf.upload(clhf, s); colAf.upload(caf, s);
      segXY.upload(sxy, s); segLH.upload(slh, s); segAr.upload(sa, s);
      segXYf.upload(sxyf, s); segLHf.upload(slhf, s); segArf.upload(saf, s);
      // extent lists: set n < NN the segments of node n, set NN the hull's columns (points ns and up; tops only)
      std::vector<std::int32_t> first(S.segStart), number(S.segCount);
      first.push_back(static_cast<std::int32_t>(ns));
      number.push_back(static_cast<std::int32_t>(nc));
      auto xy = [&](std::int32_t i) { const auto k = static_cast<std::size_t>(i); return k < ns ? sxy[k] : cxy[k - ns]; };
      auto lh = [&](std::int32_t i) { const auto k = static_cast<std::size_t>(i); return k < ns ? slh[k] : clh[k - ns]; };
      const ExtentLists lists = extent_lists(
          first, number, [&](std::int32_t i) { return xy(i).x; }, [&](std::int32_t i) { return xy(i).y; },
          [&](std::int32_t i) { return lh(i).x; }, [&](std::int32_t i) { return lh(i).y; });
      std::vector<double2> exy(lists.idx.size());
      std::vector<float2> exyf(lists.idx.size());
      std::vector<double> ez(lists.idx.size());
      std::vector<float> ezf(lists.idx.size());
      for (std::size_t l = 0; l + 1 < lists.start.size(); ++l) {
        const bool top = (l / first.size()) & 1;
        for (auto k = static_cast<std::size_t>(lists.start[l]); k < static_cast<std::size_t>(lists.start[l + 1]); ++k) {
          exy[k] = xy(lists.idx[k]);
          ez[k] = top ? lh(lists.idx[k]).y : lh(lists.idx[k]).x;
          exyf[k] = float2{static_cast<float>(exy[k].x), static_cast<float>(exy[k].y)};
          ezf[k] = static_cast<float>(ez[k]);
        }
      }
      exStart.upload(lists.start, s); exXY.upload(exy, s); exZ.upload(ez, s); exXYf.upload(exyf, s); exZf.upload(ezf, s);
      check(cudaStreamSynchronize(s), "stream sync");
    }
    mu.upload(S.mu, s); vmax.upload(S.vmax, s); amin.upload(S.amin, s); aov.upload(S.aov, s);
    std::vector<int2> ns(static_cast<std::size_t>(NN));
    for (std::size_t n = 0; n < ns.size(); ++n) ns[n] = int2{S.segStart[n], S.segCount[n]};
    nodeSeg.upload(ns, s);
    segStart.upload(S.segStart, s); segCount.upload(S.segCount, s);
    gStart.upload(M.gNodeStart, s); gCount.upload(M.gNodeCount, s); gNodes.upload(M.gNodes, s); gMode.upload(M.gMode, s);
    std::vector<Listed> entry(static_cast<std::size_t>(NG));
    for (std::size_t g = 0; g < entry.size(); ++g) {
      const std::int32_t* m = M.gNodes.data() + M.gNodeStart[g];
      const std::int32_t N = M.gNodeCount[g];
      const std::int32_t first = N > 0 ? m[0] : 0;
      entry[g] = Listed{static_cast<std::uint16_t>(g), static_cast<std::uint16_t>(first), static_cast<std::uint16_t>(N > 1 ? m[1] : first),
                        static_cast<std::uint8_t>(std::min(N, 255)), M.gMode[g]};
    }
    groupEntry.upload(entry, s);
    gpx.upload(M.gpx, s); gpy.upload(M.gpy, s); gpz.upload(M.gpz, s);
    ca.upload(M.ca, s); cb.upload(M.cb, s); skip.upload(M.cSkipGroup, s); law.upload(M.cLaw, s);
    kx.upload(M.cx, s); ky.upload(M.cy, s); kz.upload(M.cz, s); coef.upload(M.cCoef, s);
    incStart.upload(inc.start, s); incCount.upload(inc.count, s); incConn.upload(inc.conn, s); incSide.upload(inc.side, s);
    std::vector<std::int32_t> edge(inc.conn.size());
    for (std::size_t k = 0; k < edge.size(); ++k) edge[k] = 2 * inc.conn[k] + (inc.side[k] ? 1 : 0);
    incEdge.upload(edge, s);
    sea.upload(inc.sea.empty() ? std::vector<std::int32_t>{0} : inc.sea, s);
    monStart.upload(mons.start.empty() ? std::vector<std::int32_t>{0} : mons.start, s);
    monCount.upload(mons.count.empty() ? std::vector<std::int32_t>{0} : mons.count, s);
    monConn.upload(mons.conn.empty() ? std::vector<std::int32_t>{0} : mons.conn, s);
    mkx.upload(M.mkx.empty() ? std::vector<double>{0} : M.mkx, s);
    mky.upload(M.mky.empty() ? std::vector<double>{0} : M.mky, s);
    mkz.upload(M.mkz.empty() ? std::vector<double>{0} : M.mkz, s);
    mkWhen.upload(M.mkWhen.empty() ? std::vector<std::uint8_t>{0} : M.mkWhen, s);
    check(cudaStreamSynchronize(s), "model upload");

    DevModel& d = dm;
    d.ncol = S.columns();
    d.colXY = colXY.get(); d.colLH = colLH.get(); d.colA = colA.get();
    d.colXYf = colXYf.get(); d.colLHf = colLHf.get(); d.colAf = colAf.get();
    d.nseg = S.segments();
    d.segXY = segXY.get(); d.segLH = segLH.get(); d.segAr = segAr.get();
    d.segXYf = segXYf.get(); d.segLHf = segLHf.get(); d.segArf = segArf.get();
    d.exStart = exStart.get(); d.exXY = exXY.get(); d.exZ = exZ.get(); d.exXYf = exXYf.get(); d.exZf = exZf.get();
    d.nn = NN;
    d.mu = mu.get(); d.vmax = vmax.get(); d.amin = amin.get(); d.aov = aov.get();
    d.segStart = segStart.get(); d.segCount = segCount.get(); d.nodeSeg = nodeSeg.get();
    d.ng = NG;
    d.gStart = gStart.get(); d.gCount = gCount.get(); d.gNodes = gNodes.get(); d.gMode = gMode.get(); d.groupEntry = groupEntry.get();
    d.gpx = gpx.get(); d.gpy = gpy.get(); d.gpz = gpz.get(); d.gMargin = M.gMargin; d.maxGroup = maxGroup;
    d.nc = NC;
    d.ca = ca.get(); d.cb = cb.get(); d.skip = skip.get(); d.law = law.get();
    d.kx = kx.get(); d.ky = ky.get(); d.kz = kz.get(); d.coef = coef.get();
    d.incStart = incStart.get(); d.incCount = incCount.get(); d.incConn = incConn.get(); d.incSide = incSide.get(); d.incEdge = incEdge.get();
    d.nsea = static_cast<std::int32_t>(inc.sea.size()); d.sea = sea.get();
    d.nmon = nmon; d.monThreshold = M.monitorThreshold;
    d.monStart = monStart.get(); d.monCount = monCount.get(); d.monConn = monConn.get();
    d.nmark = nmark; d.mkx = mkx.get(); d.mky = mky.get(); d.mkz = mkz.get(); d.mkWhen = mkWhen.get();
    d.hullTopBelow = M.hullTopBelow; d.pitchAbsAbove = M.pitchAbsAbove; d.buoyancyBelow = M.buoyancyBelow; d.minT = M.minT;
    d.rho = M.rho; d.g = M.g; d.sq2g = std::sqrt(2 * M.g); d.dt = M.dt;
    d.ms = M.body[0]; d.g0x = M.body[2]; d.g0y = M.body[3]; d.g0z = M.body[4]; d.XO = M.body[5]; d.YO = M.body[6];
    d.mh0 = M.body[7]; d.Ith0 = M.body[8]; d.Iph0 = M.body[9]; d.cDz = M.body[10]; d.cDth = M.body[11]; d.cDph = M.body[12];
    d.qz = M.body[13]; d.qth = M.body[14]; d.qph = M.body[15];
    d.xFP = M.xFP; d.xAP = M.xAP;
    d.evCap = evCap;
  }
};

}  // namespace ssb
