"""The work a user of this engine has it do, as cases that can be timed and compared: batch runs of the compiled
titanic64 hull, of the generated liner and of mixed fleets, what-if windows in the caller's own device memory, and
gradients by the adjoint. Each case is a dict of plain values; `prepare` makes what a program holds before the call
(the batch or adjoint handle with its instances' settings), `run` is one public call with its results read back.

  batch    Batch.reset() + Batch.run(): upload, run to the end, download; then every instance's state, length and stop
  window   Batch.run_noalloc() in torch tensors: instances advance a short horizon from their current state
  adjoint  Adjoint.run(): objective, gradient with respect to every connection area, sampled trim and heave
"""
import math
import os
import tempfile

import numpy as np
import torch

import sinksim_b200 as ssb
from sinksim_b200 import hullgen
from sinksim_b200.calibrate import workload_point, workload_space
from sinksim_b200.files import decompressed, load_model
from sinksim_b200.workloads import batch_uneven, deck_edge_rule

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SAMPLES = 8          # times of an adjoint objective


def listed():
    return [
        # one simulation watched closely (the drop-in runner's trace of a single run): nothing but step latency
        {"name": "single_trace", "path": "batch", "model": "titanic64", "numerics": "portable", "count": 1, "t_max": 300.0, "curve": 10.0,
         "traced": 1, "uneven": False, "rule": False},
        # a what-if window of a control loop: a few variants half a minute ahead, in the host program's own buffers
        {"name": "window_16", "path": "window", "model": "titanic64", "numerics": "portable", "count": 16, "t_max": 30.0},
        # the same for a larger ensemble in the single-precision columns
        {"name": "window32_401", "path": "window", "model": "titanic64", "numerics": "portable32", "count": 401, "t_max": 61.0},
        # a sweep file's size and defaults (portable32, a readout curve every minute)
        {"name": "sweep32_48", "path": "batch", "model": "titanic64", "numerics": "portable32", "count": 48, "t_max": 900.0, "curve": 60.0,
         "traced": 0, "uneven": True, "rule": False},
        # runs of very different length to deep flooding: the retire rule, and the large teams of the last phases
        {"name": "long_192", "path": "batch", "model": "titanic64", "numerics": "portable", "count": 192, "t_max": 3600.0, "curve": 0.0,
         "traced": 0, "uneven": True, "rule": True},
        # the benchmark's uneven batch at half its count, to 20 min: the main phase at full load
        {"name": "uneven_2048", "path": "batch", "model": "titanic64", "numerics": "portable", "count": 2048, "t_max": 1200.0, "curve": 0.0,
         "traced": 0, "uneven": True, "rule": True},
        # the same kind of batch in portable32, an odd count
        {"name": "uneven32_1021", "path": "batch", "model": "titanic64", "numerics": "portable32", "count": 1021, "t_max": 900.0, "curve": 30.0,
         "traced": 0, "uneven": True, "rule": True},
        # perturbed copies of the liner (one space per group, twice the segments)
        {"name": "liner_264", "path": "batch", "model": "liner", "numerics": "portable", "count": 264, "t_max": 900.0, "curve": 0.0,
         "traced": 0, "uneven": True, "rule": False},
        # a mixed fleet: hulls of 1,200 to 16,600 columns and 16 to 256 spaces, several variants of each
        {"name": "fleet_12x8", "path": "fleet", "numerics": "portable", "hulls": 12, "copies": 8, "t_max": 300.0},
        # calibration on the liner: one gradient per point, 16-warp teams
        {"name": "adjoint_64", "path": "adjoint", "model": "liner", "count": 64, "t_max": 400.0},
        # more points than two per SM: 8-warp teams
        {"name": "adjoint_320", "path": "adjoint", "model": "liner", "count": 320, "t_max": 150.0},
        # a handful of points on the hull with merged spaces
        {"name": "adjoint_titanic_3", "path": "adjoint", "model": "titanic64", "count": 3, "t_max": 200.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["batch", "batch", "batch", "window", "fleet", "adjoint"])
    numerics = rng.choice(["portable", "portable", "portable32"])
    if path == "batch":
        count = _log_int(rng, 1, 2000)
        # at most about the largest listed case's instance-seconds, and its wall time for few instances
        t_max = round(math.exp(rng.uniform(math.log(60.0), math.log(min(1800.0, 1.5e6 / count)))), 2)
        model = rng.choice(["titanic64", "titanic64", "liner"])
        if model == "liner":
            count = max(1, count // 2)
        return {"path": path, "model": model, "numerics": numerics, "count": count, "t_max": t_max, "curve": rng.choice([0.0, 7.5, 60.0]),
                "traced": rng.choice([0, 0, min(2, count)]), "uneven": count > 1, "rule": rng.random() < 0.4}
    if path == "window":
        return {"path": path, "model": rng.choice(["titanic64", "liner"]), "numerics": numerics, "count": _log_int(rng, 1, 800),
                "t_max": round(math.exp(rng.uniform(math.log(5.0), math.log(90.0))), 2)}
    if path == "fleet":
        return {"path": path, "numerics": numerics, "hulls": rng.randint(2, 12), "copies": _log_int(rng, 1, 12),
                "t_max": round(rng.uniform(30.0, 300.0), 2)}
    count = _log_int(rng, 1, 400)
    return {"path": path, "model": rng.choice(["liner", "titanic64"]), "count": count,
            "t_max": round(rng.uniform(40.0, 400.0 if count <= 128 else 120.0), 2)}


# ------------------------------------------------------------------------------------------ the models on disk

def _cache():
    return os.path.join(tempfile.gettempdir(), "sinksim_b200_cases_%d" % os.getuid())


def _hull(ship_id, spec, seed):
    out = _cache()
    paths = tuple(os.path.join(out, "%s.%s.json" % (ship_id, k)) for k in ("ship", "sim"))
    if not all(os.path.exists(p) for p in paths):
        paths = hullgen.write(out, spec=spec, seed=seed, ship_id=ship_id)
    return paths


def _paths(model):
    if model == "liner":
        return _hull("liner269", None, 20261203)
    golden = os.path.join(ROOT, "tests", "golden")
    return decompressed(os.path.join(golden, "titanic64.ship.json.gz")), decompressed(os.path.join(golden, "titanic.sim.json.gz"))


_models = {}


def _model(model):
    if model not in _models:
        _models[model] = load_model(*_paths(model))
    return _models[model]


def _fleet(n):
    return [_hull("fleet%02d" % i, spec, 20261204 + i) for i, spec in enumerate(hullgen.fleet_specs(n))]


# ------------------------------------------------------------------------------------------ what a program holds

def _instances(case, seed):
    """Per instance its connection areas [count, nc] and enabled flags [count, nc]."""
    _, sim = _model(case["model"])
    area = np.tile(sim["area"], (case["count"], 1))
    en = np.tile(sim["en"], (case["count"], 1))
    if case.get("uneven", True):
        for i, (a, e) in enumerate(batch_uneven(sim, case["count"], seed=1000 + seed)):
            area[i, list(a)] = list(a.values())
            en[i, list(e)] = list(e.values())
    else:
        breach = sim["kind"] == sim["kindNames"].index("breach")
        area[:, breach] *= np.random.default_rng(seed).lognormal(0.0, 0.2)
    return area, en


def _targets(case, seed):
    """The observed trajectory of an adjoint objective: sample times, and trim and heave ramps per instance."""
    rng = np.random.default_rng([seed, 7])
    times = case["t_max"] * np.arange(1, SAMPLES + 1) / SAMPLES
    ramp = times / case["t_max"]
    n = case["count"]
    return times, rng.normal(0.3, 0.1, (n, 1)) * ramp, 10.5 + rng.normal(0.3, 0.1, (n, 1)) * ramp


def _records(case):
    """Readouts in a whole run's curve, the final ones among them; a shorter run's row is filled up with zeros."""
    return math.floor(case["t_max"] / case["curve"]) + 3 if case["curve"] > 0 else 0


def prepare(case, seed):
    if case["path"] == "fleet":
        models = _fleet(case["hulls"])
        which = [i // case["copies"] for i in range(case["hulls"] * case["copies"])]
        b = ssb.Batch.fleet(models, which, numerics=case["numerics"], t_max=case["t_max"], stop_when_stable=True)
        rng = np.random.default_rng(seed)
        for i, m in enumerate(which):
            sim = _models.setdefault(models[m], load_model(*models[m]))[1]
            breach = np.nonzero(sim["kind"] == sim["kindNames"].index("breach"))[0]
            b.set_connection_areas(i, breach, (sim["area"][breach] * rng.lognormal(0.0, 0.3))[None, :])
        return {"path": "batch", "batch": b, "count": len(which), "records": 0}
    ship_p, sim_p = _paths(case["model"])
    ship, sim = _model(case["model"])
    every = np.arange(len(sim["ca"]), dtype=np.int32)
    if case["path"] == "adjoint":
        space = workload_space(sim)
        cols, areas = space.area_matrix(np.stack([workload_point(space, i, seed=2000 + seed) for i in range(case["count"])]))
        a = ssb.Adjoint(ship_p, sim_p, count=case["count"], t_max=case["t_max"])
        a.set_connection_areas(0, cols, areas)
        a.set_objective(*_targets(case, seed))
        return {"path": "adjoint", "adjoint": a}
    area, en = _instances(case, seed)
    if case["path"] == "window":
        n = case["count"]
        dev = torch.device("cuda")
        b = ssb.Batch(ship_p, sim_p, count=1, numerics=case["numerics"], t_max=case["t_max"])
        now = {"state": np.tile(np.append(sim["state0"], 0.0), (n, 1))}
        for k in ("vol", "level", "cx", "cy", "cz"):
            now[k] = np.tile(sim[k + "0"], (n, 1))
        now = {k: torch.as_tensor(v, device=dev).contiguous() for k, v in now.items()}
        return {"path": "window", "batch": b, "count": n, "now": now, "ahead": {k: torch.empty_like(v) for k, v in now.items()},
                "en": torch.as_tensor(en, device=dev).contiguous(), "area": torch.as_tensor(area, device=dev).contiguous(),
                "t_on": torch.as_tensor(np.tile(sim["tOn"], (n, 1)), device=dev).contiguous(),
                "final": torch.empty(n, 7, dtype=torch.float64, device=dev), "steps": torch.empty(n, dtype=torch.int64, device=dev),
                "stop": torch.empty(n, dtype=torch.int32, device=dev)}
    b = ssb.Batch(ship_p, sim_p, count=case["count"], numerics=case["numerics"], t_max=case["t_max"], curve_every=case["curve"],
                  traced_instances=case["traced"], rule=deck_edge_rule(ship) if case["rule"] else None)
    b.set_connection_areas(0, every, area)
    for i, c in zip(*np.nonzero(en != sim["en"])):
        b.set_connection_enabled(int(i), int(c), bool(en[i, c]))
    return {"path": "batch", "batch": b, "count": case["count"], "records": _records(case)}


def run(state):
    if state["path"] == "adjoint":
        a = state["adjoint"]
        J, grad, steps, error, _ = a.run()
        trim, heave = a.samples()
        return {"J": J, "grad": grad, "trim": trim, "heave": heave, "steps": steps, "error": error}
    b = state["batch"]
    if state["path"] == "window":
        w = state["ahead"]
        for k, v in state["now"].items():
            w[k].copy_(v)
        b.run_noalloc(state["count"], state["en"].data_ptr(), state["area"].data_ptr(), state["t_on"].data_ptr(), w["state"].data_ptr(),
                      w["vol"].data_ptr(), w["level"].data_ptr(), w["cx"].data_ptr(), w["cy"].data_ptr(), w["cz"].data_ptr(),
                      state["final"].data_ptr(), state["steps"].data_ptr(), state["stop"].data_ptr(),
                      torch.cuda.current_stream().cuda_stream or None)
        return {**w, "final": state["final"], "steps": state["steps"], "stop": state["stop"]}
    b.reset()
    b.run()
    n = state["count"]
    ends = [b.summary(i) for i in range(n)]
    out = {"state": np.concatenate([b.state(i) for i in range(n)]), "steps": np.array([e["steps"] for e in ends]),
           "foundered": np.array([e["foundered"] for e in ends]), "final": np.stack([b.final_readouts(i) for i in range(n)])}
    if state["records"]:
        out["curve"] = np.zeros((n, state["records"], 7))
        for i in range(n):
            c = b.curve(i)
            out["curve"][i, :len(c)] = c
    return out


# ------------------------------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Inputs read and outputs written once, and the operations of the steps: 17 per hull column, 19 per segment of the
    flooded spaces (a third of them), 30 per connection, 40 per space; a gradient's reverse takes twice a step's."""
    if case["path"] == "fleet":
        sizes = [(s, m, case["copies"]) for s, m in (_models.setdefault(p, load_model(*p)) for p in _fleet(case["hulls"]))]
    else:
        sizes = [(*_model(case["model"]), case["count"])]
    nbytes = flops = 0.0
    for ship, sim, n in sizes:
        nc, nn = len(sim["ca"]), len(ship["mu"])
        steps = case["t_max"] / sim["dt"]
        if case.get("rule"):  # the settle rule ends many runs at 600 s
            steps = min(steps, 600.0 / sim["dt"] + 0.4 * max(0.0, steps - 600.0 / sim["dt"]))
        op = 17.0 * len(ship["x"]) + 19.0 * len(ship["segA"]) / 3 + 30.0 * nc + 40.0 * nn
        flops += n * steps * op * (3 if case["path"] == "adjoint" else 1)
        nbytes += n * (17.0 * nc + 2 * 8.0 * (8 + 5 * nn) + (8.0 * nc if case["path"] == "adjoint" else 0))
        nbytes += 40.0 * (len(ship["x"]) + len(ship["segA"]))
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------------------ the same step in plain numpy

class _Plain:
    """One instance stepped in float64 numpy (the engine's physics: buoyancy of the clipped hull columns, the spaces'
    free-surface levels by bracketed Newton, orifice and weir flows with the limiter, loads, semi-implicit rigid body)."""

    def __init__(self, ship, sim, area, en):
        self.s, self.m, self.area, self.en = ship, sim, area, en.astype(bool)
        s, m = ship, sim
        nn = self.nn = len(s["mu"])
        self.node = np.repeat(np.arange(nn), s["segCount"])
        seg = np.concatenate([np.arange(a, a + c) for a, c in zip(s["segStart"], s["segCount"])])
        col = s["segCol"][seg]
        self.sx, self.sy, self.sA, self.sa, self.sb = s["x"][col], s["y"][col], s["dxdy"][col], s["segA"][seg], s["segE"][seg]
        self.first = np.concatenate([[0], np.cumsum(s["segCount"])[:-1]])
        self.groups = [m["gNodes"][a:a + c] for a, c in zip(m["gStart"], m["gCount"])]
        self.t, self.zO, self.th, self.ph, self.vz, self.wth, self.wph = m["state0"]
        self.vol, self.level = m["vol0"].copy(), m["level0"].copy()
        self.c = np.stack([m["cx0"], m["cy0"], m["cz0"]])
        self.inflow = self.Vb = self.top = 0.0
        self.pose()

    def pose(self):
        ct, st, cp, sp = math.cos(self.th), math.sin(self.th), math.cos(self.ph), math.sin(self.ph)
        self.R = np.array([[ct, st * sp, st * cp], [0, cp, -sp], [-st, ct * sp, ct * cp]])
        self.ct = ct
        b = self.m["body"]
        self.T = np.array([b[5], b[6], self.zO]) - self.R @ np.array(b[2:5])

    def z(self, x, y, z):
        return self.R[2, 0] * x + self.R[2, 1] * y + self.R[2, 2] * z + self.T[2]

    def readouts(self):
        rho, m = self.m["rho"], self.m
        return np.array([self.t, math.degrees(self.th), math.degrees(self.ph), self.vol.sum() * rho / 1000, self.inflow * rho / 1000 * 60,
                         -self.z(m["xFP"], 0, 0), -self.z(m["xAP"], 0, 0)])

    def record(self):
        head = [self.t, self.zO, self.th, self.ph, self.vz, self.wth, self.wph, self.inflow, self.Vb, self.top]
        return np.concatenate([head, self.vol, self.level, *self.c])

    def sum_nodes(self, v):
        return np.bincount(self.node, v, self.nn)

    def wet(self, base, h):
        zp = (h[self.node] - base) / self.R[2, 2]
        L = np.where(zp <= self.sa, 0.0, np.where(zp >= self.sb, self.sb - self.sa, zp - self.sa))
        cut = (zp > self.sa) & (zp < self.sb)
        mu = self.s["mu"]
        return self.sA * L, L, self.sum_nodes(self.sA * L) * mu, self.sum_nodes(self.sA * cut) * mu / self.R[2, 2]

    def levels(self):
        s, m = self.s, self.m
        base = self.R[2, 0] * self.sx + self.R[2, 1] * self.sy + self.T[2]
        zmin = np.minimum.reduceat(base + self.R[2, 2] * self.sa, self.first)
        self.zmax = np.maximum.reduceat(base + self.R[2, 2] * self.sb, self.first)
        self.merged = np.zeros(len(self.groups), dtype=bool)
        units = []
        for g, nodes in enumerate(self.groups):
            if len(nodes) > 1 and m["gMode"][g] == 1:
                self.merged[g] = True
            elif len(nodes) > 1 and m["gMode"][g] == 2:
                over = self.z(m["gpx"][g], m["gpy"][g], m["gpz"][g]) + m["gMargin"]
                self.merged[g] = np.all((self.vol[nodes] > 1e-6) & (self.level[nodes] > over))
            units += [nodes] if self.merged[g] else [nodes[k:k + 1] for k in range(len(nodes))]
        h = np.zeros(self.nn)
        area = np.zeros(self.nn)
        todo, final = [], np.zeros(self.nn, dtype=bool)
        for u in units:
            V, vmax = self.vol[u].sum(), s["vmax"][u].sum()
            lo, hi = zmin[u].min(), self.zmax[u].max()
            if V <= 1e-6:
                if len(u) > 1:
                    self.vol[u] = 0
                self.level[u] = zmin[u]
                continue
            final[u] = True
            if V >= vmax * (1 - 1e-7):
                dh = max(0.0, V - vmax) / s["aov"][u].sum()
                if len(u) > 1:
                    self.vol[u[:-1]] = s["vmax"][u[:-1]] + dh * s["aov"][u[:-1]]
                    self.vol[u[-1]] = V - self.vol[u[:-1]].sum()
                h[u], self.level[u], area[u] = hi, hi + dh, s["aov"][u]
                continue
            damp = self.vol[u] > 0
            start = self.level[u].mean() if damp.all() else self.level[u[int(np.argmax(damp)) if damp.any() else len(u) - 1]]
            h[u] = min(hi, max(lo, start))
            todo.append([u, V, max(1e-3 * vmax, 0.5), lo, hi, True])
        for it in range(7):
            v, L, vol, dv = self.wet(base, h)
            if it == 6 or not any(q[5] for q in todo):
                break
            for q in todo:
                u, V, tol, a, b, live = q
                if not live:
                    continue
                err, slope, at = vol[u].sum() - V, dv[u].sum(), h[u[0]]
                if abs(err) < tol:
                    q[5] = False
                    continue
                q[4 if err > 0 else 3] = at
                nxt = at - err / slope if slope > 1e-9 else 0.5 * (q[3] + q[4])
                h[u] = nxt if q[3] < nxt < q[4] else 0.5 * (q[3] + q[4])
        for u, V, *_ in todo:
            if len(u) > 1:
                share = V * vol[u] / vol[u].sum() if vol[u].sum() > 0 else np.full(len(u), V / len(u))
                share[:-1] = np.minimum(share[:-1], s["vmax"][u[:-1]])
                share[-1] = V - share[:-1].sum()
                for k in range(len(u) - 1, 0, -1):  # an overfull last member passes its surplus down
                    over = share[k] - s["vmax"][u[k]]
                    if over > 0:
                        share[k] -= over
                        share[k - 1] += over
                self.vol[u] = share
            self.level[u], area[u] = h[u], dv[u]
        mu = s["mu"]
        keep = final & (vol > 1e-9)
        for k, w in enumerate((v * self.sx, v * self.sy, v * (self.sa + 0.5 * L))):
            self.c[k, keep] = (self.sum_nodes(w) * mu)[keep] / vol[keep]
        return area

    def step(self):
        s, m = self.s, self.m
        dt, R, T = m["dt"], self.R, self.T
        base = R[2, 0] * s["x"] + R[2, 1] * s["y"] + T[2]
        self.top = (base + R[2, 2] * s["zhi"]).max()
        w = np.clip(np.minimum(-base / R[2, 2], s["zhi"]) - s["zlo"], 0, None)
        v = s["dxdy"] * w
        V = self.Vb = v.sum()
        cb = np.array([(v * s["x"]).sum(), (v * s["y"]).sum(), (v * (s["zlo"] + 0.5 * w)).sum()]) / (V if V > 0 else 1.0)
        area = self.levels()
        # flows
        wet = self.vol > 1e-6
        head = np.append(np.where(wet, self.level, -1e9), 0.0)
        inv = np.append(1 / np.where(self.vol >= s["vmax"], s["aov"], np.maximum(area, s["amin"])), 0.0)
        a, b = m["ca"], m["cb"]
        counted = self.en & ~((a >= 0) & (head[a] < -1e8) & (head[b] < -1e8))
        deg = np.bincount(a[counted & (a >= 0)], minlength=self.nn) + np.bincount(b[counted], minlength=self.nn)
        deg = np.append(deg, 0)
        on = self.en & (m["tOn"] <= self.t) & ~((m["skipGroup"] >= 0) & self.merged[m["skipGroup"]])
        zo = self.z(m["cx"], m["cy"], m["cz"])
        Ha, Hb = np.maximum(head[a] - zo, 0), np.maximum(head[b] - zo, 0)
        d, H1, H2 = Ha - Hb, np.maximum(Ha, Hb), np.minimum(Ha, Hb)
        r = np.where(H1 > 0, H2 / np.where(H1 > 0, H1, 1), 0)
        k = m["coef"] * self.area * math.sqrt(2 * m["g"])
        weir = k * (2 / 3) * H1 * np.sqrt(H1) * np.maximum(0, 1 - r ** 1.5) ** 0.385 * np.where(Ha >= Hb, 1, -1)
        q = np.where(on, np.where(m["law"] == 0, k * d / np.sqrt(np.maximum(np.abs(d), 0.01)), weir), 0) * dt
        src, dst = np.where(q > 0, a, b), np.where(q > 0, b, a)
        share = 0.5 / np.maximum(1, np.maximum(deg[src], deg[dst]))
        both = inv[src] + inv[dst]
        lim = np.maximum(0, np.where(both > 0, share * (head[src] - np.maximum(head[dst], zo)) / np.where(both > 0, both, 1), np.abs(q)))
        q = np.sign(q) * np.minimum(np.abs(q), lim)
        vol = self.vol + np.bincount(b, q, self.nn) - np.bincount(a[a >= 0], q[a >= 0], self.nn)
        vol = np.maximum(vol, 0)
        cap = s["vmax"] + s["aov"] * np.maximum(0, -self.zmax)
        excess = np.where((vol > s["vmax"]) & (vol > cap), vol - cap, 0)
        self.vol = vol - excess
        self.inflow = (q[a < 0].sum() - excess.sum()) / dt
        # loads and the rigid body
        ms, _, _, _, _, X, Y, mh, Ith, Iph, cz, cth, cph, qz, qth, qph = m["body"]
        rho, g = m["rho"], m["g"]
        F = rho * g * V
        bw = R @ cb + T
        W = R @ self.c + T[:, None] - np.array([X, Y, self.zO])[:, None]
        mass = rho * self.vol
        tauX = (bw[1] - Y) * F - (W[1] * mass).sum() * g
        tauY = -(bw[0] - X) * F + (W[0] * mass).sum() * g
        az = (F - g * ms - g * mass.sum() - cz * self.vz - qz * abs(self.vz) * self.vz) / (mh + mass.sum())
        ath = (tauY - cth * self.wth - qth * abs(self.wth) * self.wth) / (Ith + (mass * (W[0] ** 2 + W[2] ** 2)).sum())
        aph = (tauX * self.ct - cph * self.wph - qph * abs(self.wph) * self.wph) / (Iph + (mass * (W[1] ** 2 + W[2] ** 2)).sum())
        self.vz += az * dt
        self.wth += ath * dt
        self.wph += aph * dt
        self.zO += self.vz * dt
        self.th += self.wth * dt
        self.ph += self.wph * dt
        self.t += dt
        self.pose()


def exact(case, seed):
    """The small batch and window cases and the small adjoint's objective in float64 numpy (about 2 ms a step); a
    gradient, a fleet or a long batch would take far longer than 20 s this way."""
    if case["path"] == "fleet" or case.get("rule"):
        return None
    ship, sim = _model(case["model"])
    if case["count"] * case["t_max"] / sim["dt"] * len(ship["segA"]) / 8706 > 4000:
        return None
    if case["path"] == "adjoint":
        space = workload_space(sim)
        cols, areas = space.area_matrix(np.stack([workload_point(space, i, seed=2000 + seed) for i in range(case["count"])]))
        area, en = np.tile(sim["area"], (case["count"], 1)), np.tile(sim["en"], (case["count"], 1))
        area[:, cols] = areas
        times, trim_t, heave_t = _targets(case, seed)
        trim, heave = np.empty_like(trim_t), np.empty_like(heave_t)
    else:
        area, en = _instances(case, seed)
    states, finals, curves = [], [], []
    for i in range(case["count"]):
        p = _Plain(ship, sim, area[i], en[i])
        k, next_curve, curve = 0, 0.0, []
        while True:
            done = p.t >= case["t_max"]
            if case["path"] == "adjoint":
                while k < SAMPLES and (done or p.t >= times[k]):
                    r = p.readouts()
                    trim[i, k], heave[i, k] = r[1], 0.5 * (r[5] + r[6])
                    k += 1
            if done:
                break
            if case.get("curve") and p.t >= next_curve:
                curve.append(p.readouts())
                next_curve += case["curve"]
            p.step()
        states.append(p.record())
        finals.append(p.readouts())
        curves.append(curve + [p.readouts()])
    if case["path"] == "adjoint":
        J = ((trim - trim_t) ** 2 + (heave - heave_t) ** 2).sum(1)
        return {"J": J, "grad": None, "trim": trim, "heave": heave, "steps": None, "error": None}
    if case["path"] == "window":
        r, n = np.stack(states), len(ship["mu"])
        out = {"state": np.concatenate([r[:, :7], np.zeros((len(r), 1))], 1), "final": np.stack(finals), "steps": None, "stop": None}
        for j, k in enumerate(("vol", "level", "cx", "cy", "cz")):
            out[k] = r[:, 10 + j * n:10 + (j + 1) * n].copy()
        return out
    out = {"state": np.concatenate(states), "steps": None, "foundered": None, "final": np.stack(finals)}
    if case["curve"] > 0:
        out["curve"] = np.zeros((case["count"], _records(case), 7))
        for row, c in zip(out["curve"], curves):
            row[:len(c)] = c
    return out
