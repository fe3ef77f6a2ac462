// Device memory of one compiled model and of the buffers the engines own: DevBuf (an owning device array) and ModelDev
// (a compiled ship and sim in the kernels' layout, DevModel pointing into it). Shared by the batch engine (batch.cpp)
// and the adjoint engine (adjoint.cpp).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

#include "device_model.h"
#include "extents.h"
#include "model.h"
#include "slot_layout.h"

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

// Tables of one model put together on the host and copied to the device in one piece (a model has some fifty, and an
// allocation and a copy of each cost more than building them); every table starts at a multiple of 256 bytes.
class TablePack {
 public:
  template <class T>
  void add(const T*& slot, const std::vector<T>& v) {
    const std::size_t at = (host_.size() + 255) & ~static_cast<std::size_t>(255);
    host_.resize(at + std::max<std::size_t>(v.size() * sizeof(T), 1));
    if (!v.empty()) std::memcpy(host_.data() + at, v.data(), v.size() * sizeof(T));
    places_.push_back({reinterpret_cast<const void**>(&slot), at});
  }
  // Copies the tables into `to` and points the slots at them.
  void upload(DevBuf<unsigned char>& to, cudaStream_t s) {
    to.upload(host_, s);
    check(cudaStreamSynchronize(s), "model upload");
    for (const auto& p : places_) *p.first = to.get() + p.second;
  }

 private:
  std::vector<unsigned char> host_;
  std::vector<std::pair<const void**, std::size_t>> places_;
};

// One compiled model on the device: its geometry in the kernel's layout (paired fields, the segment -> column gather
// resolved, float copies), its node, group, connection, incidence, monitor and mark tables, and the DevModel that
// points into them.
struct ModelDev {
  std::shared_ptr<const CompiledShip> ship;
  CompiledSim sim;
  Incidence inc;
  MonitorLists mons;
  std::int32_t NN = 0, NC = 0, NG = 0, nmon = 0, nmark = 0, evCap = 0, maxGroup = 0;
  DevBuf<unsigned char> tables;
  DevModel dm{};

  ModelDev(std::shared_ptr<const CompiledShip> s, const CompiledSim& m) : ship(std::move(s)), sim(m) {
    if (!ship) throw std::invalid_argument("Batch: null ship");
    check_pairing(*ship, sim);
    inc = build_incidence(sim);
    mons = build_monitor_lists(sim);
    NN = ship->nodes(); NC = sim.connections(); NG = sim.groups();
    nmon = sim.monitors(); nmark = sim.marks(); evCap = nmon + nmark + 1; maxGroup = sim.maxGroupSize();
    if (NG >= 32768) throw std::runtime_error("simulation " + sim.id + " has " + std::to_string(NG) + " groups, the level solve lists up to 32767");
  }

  void upload(cudaStream_t s) {
    const CompiledShip& S = *ship;
    DevModel& d = dm;
    TablePack pack;
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
      pack.add(d.colXY, cxy); pack.add(d.colLH, clh); pack.add(d.colA, S.dxdy);
      pack.add(d.colXYf, cxyf); pack.add(d.colLHf, clhf); pack.add(d.colAf, caf);
      pack.add(d.segXY, sxy); pack.add(d.segLH, slh); pack.add(d.segAr, sa);
      pack.add(d.segXYf, sxyf); pack.add(d.segLHf, slhf); pack.add(d.segArf, saf);
      // extent lists: set n < NN the segments of node n, set NN the hull's columns (points ns and up; tops only)
      std::vector<std::int32_t> first(S.segStart), number(S.segCount);
      first.push_back(static_cast<std::int32_t>(ns));
      number.push_back(static_cast<std::int32_t>(nc));
      auto xy = [&](std::int32_t i) { const auto k = static_cast<std::size_t>(i); return k < ns ? sxy[k] : cxy[k - ns]; };
      auto lh = [&](std::int32_t i) { const auto k = static_cast<std::size_t>(i); return k < ns ? slh[k] : clh[k - ns]; };
      const ExtentLists lists = extent_lists(
          first, number, [&](std::int32_t i) { return xy(i).x; }, [&](std::int32_t i) { return xy(i).y; },
          [&](std::int32_t i) { return lh(i).x; }, [&](std::int32_t i) { return lh(i).y; },
          static_cast<std::size_t>(NN));
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
      pack.add(d.exStart, lists.start); pack.add(d.exXY, exy); pack.add(d.exZ, ez); pack.add(d.exXYf, exyf); pack.add(d.exZf, ezf);
    }
    pack.add(d.mu, S.mu); pack.add(d.vmax, S.vmax); pack.add(d.amin, S.amin); pack.add(d.aov, S.aov);
    std::vector<int2> ns(static_cast<std::size_t>(NN));
    for (std::size_t n = 0; n < ns.size(); ++n) ns[n] = int2{S.segStart[n], S.segCount[n]};
    pack.add(d.nodeSeg, ns);
    pack.add(d.segStart, S.segStart); pack.add(d.segCount, S.segCount);
    pack.add(d.gStart, M.gNodeStart); pack.add(d.gCount, M.gNodeCount); pack.add(d.gNodes, M.gNodes);
    std::vector<GroupEntry> entry(static_cast<std::size_t>(NG));
    for (std::size_t g = 0; g < entry.size(); ++g) {
      const std::int32_t* m = M.gNodes.data() + M.gNodeStart[g];
      const std::int32_t N = M.gNodeCount[g];
      const std::int32_t first = N > 0 ? m[0] : 0;
      entry[g] = GroupEntry{static_cast<std::uint16_t>(first), static_cast<std::uint16_t>(N > 1 ? m[1] : first),
                            static_cast<std::uint8_t>(std::min(N, 255)), M.gMode[g]};
    }
    pack.add(d.groupEntry, entry);
    pack.add(d.gpx, M.gpx); pack.add(d.gpy, M.gpy); pack.add(d.gpz, M.gpz);
    pack.add(d.ca, M.ca); pack.add(d.cb, M.cb); pack.add(d.skip, M.cSkipGroup); pack.add(d.law, M.cLaw);
    pack.add(d.kx, M.cx); pack.add(d.ky, M.cy); pack.add(d.kz, M.cz); pack.add(d.coef, M.cCoef);
    pack.add(d.incStart, inc.start); pack.add(d.incCount, inc.count); pack.add(d.incConn, inc.conn); pack.add(d.incSide, inc.side);
    std::vector<std::int32_t> edge(inc.conn.size());
    for (std::size_t k = 0; k < edge.size(); ++k) edge[k] = 2 * inc.conn[k] + (inc.side[k] ? 1 : 0);
    pack.add(d.incEdge, edge);
    pack.add(d.sea, inc.sea.empty() ? std::vector<std::int32_t>{0} : inc.sea);
    pack.add(d.monStart, mons.start.empty() ? std::vector<std::int32_t>{0} : mons.start);
    pack.add(d.monCount, mons.count.empty() ? std::vector<std::int32_t>{0} : mons.count);
    pack.add(d.monConn, mons.conn.empty() ? std::vector<std::int32_t>{0} : mons.conn);
    pack.add(d.mkx, M.mkx.empty() ? std::vector<double>{0} : M.mkx);
    pack.add(d.mky, M.mky.empty() ? std::vector<double>{0} : M.mky);
    pack.add(d.mkz, M.mkz.empty() ? std::vector<double>{0} : M.mkz);
    pack.add(d.mkWhen, M.mkWhen.empty() ? std::vector<std::uint8_t>{0} : M.mkWhen);
    pack.upload(tables, s);

    d.ncol = S.columns(); d.nseg = S.segments(); d.nn = NN; d.ng = NG; d.nc = NC;
    d.gMargin = M.gMargin; d.maxGroup = maxGroup;
    d.nsea = static_cast<std::int32_t>(inc.sea.size());
    d.nmon = nmon; d.monThreshold = M.monitorThreshold; d.nmark = nmark;
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
