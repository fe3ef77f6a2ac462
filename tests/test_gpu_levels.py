"""The level solve over the listed groups with extent lists (csrc/warp_step.cuh) against the C restatement, from restored
states that put the spaces at the edges of its cases: dry, below the empty volume, partly flooded with the level inside
and outside the space, full, overfull; upright, heeled and beyond a quarter turn."""
import json

import numpy as np
import pytest

import sinksim_b200 as ssb
from _support import Oracle, load_model, titanic
from sinksim_b200 import hullgen

pytestmark = pytest.mark.gpu

STEPS = 12


def _records(ship, sim):
    rng = np.random.default_rng(20261206)
    nn = len(ship["mu"])
    t0, zO = sim["state0"][0], sim["state0"][1]
    for pitch, roll in ((0.0, 0.0), (0.02, 0.0), (-0.03, 0.2), (0.4, -0.5), (2.0, 0.3), (-0.1, -1.9)):
        case = rng.integers(0, 7, nn)
        vol = np.choose(case, [np.zeros(nn), np.full(nn, 7e-7), 0.3 * ship["vmax"], 0.7 * ship["vmax"], ship["vmax"], 1.02 * ship["vmax"],
                               np.full(nn, 0.4)])
        level = sim["level0"] + rng.uniform(-3.0, 6.0, nn)
        rec = np.concatenate([[t0, zO + rng.uniform(-1, 1), pitch, roll, 0.01, 1e-3, -1e-3, 0, 0, 0], vol, level, sim["cx0"], sim["cy0"], sim["cz0"]])
        yield rec


def _grouped_liner(out):
    """The generated liner with its spaces in groups of 3, 1, 4 and 2, always merged or merged above a sill by turns."""
    ship_p, sim_p = hullgen.write(out)
    sim = json.load(open(sim_p))
    n, start, count, mode = len(sim["state0"]["vol"]), [], [], []
    while sum(count) < n:
        start.append(sum(count))
        count.append(min((3, 1, 4, 2)[len(count) % 4], n - sum(count)))
        mode.append(1 + len(mode) % 2)
    g = len(count)
    sim["groups"] = dict(sim["groups"], n=g, nodeStart=start, nodeCount=count, mode=mode, px=[0.0] * g, py=[0.0] * g, pz=[4.0] * g)
    kinds = dict(nodeStart="i32", nodeCount="i32", nodes="i32", mode="u8", a="i32", b="i32", type="u8", kind="u8", idx="i32", en="u8", skipGroup="i32",
                 monitor="i32", when="u8")
    order = [("groups", ("nodeStart", "nodeCount", "nodes", "mode", "px", "py", "pz")),
             ("connections", ("a", "b", "type", "x", "y", "z", "area", "coef", "kind", "idx", "en", "tOn", "skipGroup", "monitor")),
             ("marks", ("x", "y", "z", "when")), ("state0", ("vol", "level", "cx", "cy", "cz"))]
    sim["hash"] = hullgen.hash_arrays([(f"{part}.{k}", kinds.get(k, "f64"), sim[part][k]) for part, keys in order for k in keys])
    with open(sim_p, "w") as f:
        json.dump(sim, f)
    return ship_p, sim_p


@pytest.mark.parametrize("warps", [1, 2, 8, 16])
@pytest.mark.parametrize("numerics,mixed", [("portable", False), ("portable32", True)])
@pytest.mark.parametrize("model", ["titanic64", "liner", "grouped"])
def test_restored_states_step_like_the_restatement(tmp_path, model, numerics, mixed, warps):
    ship_p, sim_p = titanic() if model == "titanic64" else (hullgen.write if model == "liner" else _grouped_liner)(str(tmp_path))
    ship, sim = load_model(ship_p, sim_p)
    records = list(_records(ship, sim))
    b = ssb.Batch(ship_p, sim_p, count=len(records), numerics=numerics, t_max=STEPS * sim["dt"], team_warps=warps, tail_team_warps=0,
                  traced_instances=len(records), dense_steps=STEPS)
    for i, r in enumerate(records):
        b.restore(i, r)
    b.run()
    for i, r in enumerate(records):
        o = Oracle(ship, sim, mixed)
        o.restore(r)
        while not o.foundered()[0] and o.record()[0] < STEPS * sim["dt"]:
            o.step(1)
        np.testing.assert_array_equal(b.state(i), o.record(), err_msg=f"record {i}")
    b.close()
