"""The two forms of a unit's reverse (sinksim_b200/csrc/adjoint_step.cuh) on the CPU: single_reverse, for a space alone that
is empty, full or solved by Newton steps, gives the bits of unit_reverse, the general form, on the units of steps recorded
by the C restatement from states at the edges of the level solve's cases."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from _support import REF_DIR, ROOT, _p, _Ship, _Sim, _structs, load_model, titanic

SOURCE = r"""
#include "adjoint_host.cpp"
#include <random>
/* Steps the model from `record` and reverses every plain single unit of every step in both forms, with random adjoints of
 * its solved values (some of them zero). seen counts the units by kind: empty, full, solved by 0 or by more Newton steps,
 * started at the space's bottom or top. Returns the number of units whose results differ in any bit. */
extern "C" int compare_units(const sso_ship* ship, const sso_sim* sim, const double* record, int steps, int64_t* seen) {
  HostModel hm(ship, sim);
  const DevModel& M = hm.dm;
  const int nn = M.nn, R = 10 + 5 * nn;
  sso_engine* e = sso_create(ship, sim, 0);
  sso_restore(e, record);
  Recorder rec{e, tape_layout(nn, M.ng), nn, M.ng};
  sso_set_hooks(e, &Recorder::on_pass, &Recorder::on_solved, &rec);
  std::mt19937_64 g(20261207);
  std::normal_distribution<double> normal;
  std::vector<double> r(static_cast<std::size_t>(R));
  int wrong = 0;
  for (int s = 0; s < steps; ++s) {
    std::vector<unsigned char> mem(rec.L.bytes, 0);
    Tape t = tape_at(mem.data(), rec.L);
    sso_get_record(e, r.data());
    for (int n = 0; n < nn; ++n) {
      t.d[rec.L.volIn + n] = r[10 + n]; t.d[rec.L.levelIn + n] = r[10 + nn + n];
      t.d[rec.L.cxIn + n] = r[10 + 2 * nn + n]; t.d[rec.L.cyIn + n] = r[10 + 3 * nn + n]; t.d[rec.L.czIn + n] = r[10 + 4 * nn + n];
    }
    rec.cur = &mem;
    sso_step(e, 1);
    const PoseD F = load_pose(t.d + rec.L.pose);
    for (int q = 0; q < M.ng; ++q) {
      if (t.i[rec.L.merged + q]) continue;
      for (int k = 0; k < M.gCount[q]; ++k) {
        const int* member = M.gNodes + M.gStart[q] + k;
        Replay p{};
        replay_unit(M, t, member, 1, true, p);
        if (!p.ok || !is_plain_single(p)) continue;
        seen[p.cs == 0 ? 0 : p.cs == 1 ? 1 : p.K == p.base ? 2 : 3]++;
        if (p.cs == 2 && p.base == 1) seen[4]++;
        double in[7], one[5];
        for (double& v : in) v = g() % 5 == 0 ? 0.0 : normal(g);
        AdjPose pa, pb;
        zero(pa);
        for (int f = 0; f < kAdjPoseFields; ++f) fields(pa)[f] = normal(g);
        pb = pa;
        static UnitWork w, v;
        single_reverse(M, F, t, p, w, in, one, 0, 1, pa);
        v.r = p;
        v.u.aLevel[0] = in[0]; v.u.aArea[0] = in[1]; v.u.aCx[0] = in[2]; v.u.aCy[0] = in[3]; v.u.aCz[0] = in[4]; v.u.aVol[0] = in[5]; v.u.aZmax[0] = in[6];
        int err = 0;
        const bool done = unit_reverse(M, F, t, v, 0, 1, pb, &err);
        const double two[5] = {v.u.oVol[0], v.u.oLevel[0], v.u.oCx[0], v.u.oCy[0], v.u.oCz[0]};
        wrong += !done || err || std::memcmp(one, two, sizeof one) || std::memcmp(&pa, &pb, sizeof pa);
      }
    }
  }
  sso_set_hooks(e, nullptr, nullptr, nullptr);
  sso_destroy(e);
  return wrong;
}
"""


@pytest.fixture(scope="module")
def compare(tmp_path_factory):
    out = tmp_path_factory.mktemp("units")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    (out / "units.cpp").write_text(SOURCE)
    oracle = os.path.join(ROOT, "oracle")
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-w", "-I", include, "-I", oracle,
                    str(out / "units.cpp"), os.path.join(REF_DIR, "libsinksim_oracle.so"), f"-Wl,-rpath,{REF_DIR}", "-o", str(out / "units.so")],
                   check=True)
    lib = C.CDLL(str(out / "units.so"))
    lib.compare_units.argtypes = [C.POINTER(_Ship), C.POINTER(_Sim), C.POINTER(C.c_double), C.c_int, C.POINTER(C.c_int64)]
    return lib.compare_units


def _records(ship, sim):
    rng = np.random.default_rng(20261208)
    nn = len(ship["mu"])
    for pitch, roll in ((0.0, 0.0), (-0.03, 0.2), (0.4, -0.5), (2.0, 0.3)):
        vol = np.choose(rng.integers(0, 7, nn), [np.zeros(nn), np.full(nn, 7e-7), 0.3 * ship["vmax"], 0.7 * ship["vmax"], ship["vmax"],
                                                 1.02 * ship["vmax"], np.full(nn, 0.4)])
        level = sim["level0"] + rng.uniform(-3.0, 6.0, nn)
        yield np.concatenate([[0.0, sim["state0"][1] + rng.uniform(-1, 1), pitch, roll, 0.01, 1e-3, -1e-3, 0, 0, 0], vol, level, sim["cx0"],
                              sim["cy0"], sim["cz0"]])


@pytest.mark.parametrize("model", ["titanic64", "liner"])
def test_single_reverse_equals_unit_reverse(compare, tmp_path, model):
    from sinksim_b200 import hullgen

    ship, sim = load_model(*(titanic() if model == "titanic64" else hullgen.write(str(tmp_path))))
    S, M = _structs(ship, sim)
    seen = np.zeros(5, dtype=np.int64)
    for rec in _records(ship, sim):
        assert compare(C.byref(S), C.byref(M), _p(rec, C.c_double), 12, _p(seen, C.c_int64)) == 0
    # (titanic64's spaces are mostly merged groups; the liner's are all alone)
    assert (seen[[0, 1, 3]] > 0).all() and (model == "titanic64" or (seen > 0).all()), seen
