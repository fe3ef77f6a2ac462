"""Models whose spaces share free surfaces in groups of more than two. In large groups the engine picks team sizes whose
pass buffers fit, and steps them like the C restatement. The adjoint's recorded steps of groups of one to four, from states
at the edges of the level solve's cases, give the host adjoint's objective bit for bit and its gradients within 1e-9 (the
device adds the pose's adjoints in another order), whether they are recorded on the way or recomputed."""
import json

import numpy as np
import pytest

import sinksim_b200 as ssb
import test_gpu_levels as levels
from _support import Oracle, adjoint_host_gradient, load_model
from sinksim_b200 import hullgen

pytestmark = pytest.mark.gpu

STEPS = 8


def _regrouped(out, counts, modes, spec=None, state0=None):
    """A generated hull with its spaces in groups of counts[0], counts[1], ... by turns (the last one cut short), and state0's
    values in place of the compiled ones."""
    ship_p, sim_p = hullgen.write(out, spec=spec)
    ship, arrays = load_model(ship_p, sim_p)
    sim = json.load(open(sim_p))
    n, start, count, mode = len(sim["state0"]["vol"]), [], [], []
    while sum(count) < n:
        start.append(sum(count))
        mode.append(modes[len(count) % len(modes)])
        count.append(min(counts[len(count) % len(counts)], n - start[-1]))
    g = len(count)
    sim["groups"] = dict(sim["groups"], n=g, nodeStart=start, nodeCount=count, mode=mode, px=[0.0] * g, py=[0.0] * g, pz=[4.0] * g)
    sim["connections"]["skipGroup"] = [-1] * sim["connections"]["n"]
    sim["state0"].update(state0(ship, arrays) if state0 else {})
    kinds = dict(nodeStart="i32", nodeCount="i32", nodes="i32", mode="u8", a="i32", b="i32", type="u8", kind="u8", idx="i32", en="u8", skipGroup="i32",
                 monitor="i32", when="u8")
    order = [("groups", ("nodeStart", "nodeCount", "nodes", "mode", "px", "py", "pz")),
             ("connections", ("a", "b", "type", "x", "y", "z", "area", "coef", "kind", "idx", "en", "tOn", "skipGroup", "monitor")),
             ("marks", ("x", "y", "z", "when")), ("state0", ("vol", "level", "cx", "cy", "cz"))]
    sim["hash"] = hullgen.hash_arrays([(f"{part}.{k}", kinds.get(k, "f64"), sim[part][k]) for part, keys in order for k in keys])
    with open(sim_p, "w") as f:
        json.dump(sim, f)
    return ship_p, sim_p


@pytest.mark.parametrize("numerics,mixed", [("portable", False), ("portable32", True)])
@pytest.mark.parametrize("spaces", [184, 256])
def test_a_group_too_large_for_the_largest_teams_runs(tmp_path, numerics, mixed, spaces):
    spec = next(s for s in hullgen.fleet_specs(12) if s.n_comp * s.n_decks == spaces)
    ship_p, sim_p = _regrouped(str(tmp_path), (spaces,), (1,), spec)
    ship, sim = load_model(ship_p, sim_p)
    with ssb.Batch(ship_p, sim_p, count=3, numerics=numerics, t_max=STEPS * sim["dt"]) as b:
        b.run()
        o = Oracle(ship, sim, mixed)
        o.step(STEPS)
        for i in range(3):
            np.testing.assert_array_equal(b.state(i), o.record(), err_msg=f"instance {i}")
    if not mixed:  # 16 warps, each with two lane groups of 40-byte passes
        for asked in (dict(team_warps=16), dict(team_warps=8, tail_team_warps=16)):
            with pytest.raises(RuntimeError, match="16-warp simulation needs more shared memory"):
                ssb.Batch(ship_p, sim_p, count=3, numerics=numerics, t_max=STEPS * sim["dt"], **asked)


@pytest.mark.parametrize("numerics,mixed", [("portable", False), ("portable32", True)])
@pytest.mark.parametrize("model", ["titanic64", "liner", "grouped"])
def test_restored_states_in_four_warp_teams(tmp_path, model, numerics, mixed):
    levels.test_restored_states_step_like_the_restatement(tmp_path, model, numerics, mixed, 4)


def _edge_state(pitch, roll, full):
    def state(ship, sim):
        rng = np.random.default_rng(20261209)
        nn = len(ship["mu"])
        share = 1.0 if full else 0.1  # (little water leaves no member of a group overfull)
        vol = np.choose(rng.integers(0, 7, nn) if full else rng.choice([0, 1, 2, 3, 6], nn),
                        [np.zeros(nn), np.full(nn, 7e-7), 0.3 * share * ship["vmax"], 0.7 * share * ship["vmax"], ship["vmax"], 1.02 * ship["vmax"],
                         np.full(nn, 0.4)])
        return dict(pitch=pitch, roll=roll, vol=vol.tolist(), level=(sim["level0"] + rng.uniform(-3.0, 6.0, nn)).tolist())

    return state


@pytest.mark.parametrize("warps", [4, 8, 16])
@pytest.mark.parametrize("pitch,roll", [(0.0, 0.0), (-0.03, 0.2), (0.1, -0.5)])
@pytest.mark.parametrize("counts,full", [((3, 1, 4, 2), True), ((3, 1, 4, 2), False), ((1,), True)], ids=["groups", "unfilled-groups", "alone"])
def test_gradients_from_edge_states(tmp_path, counts, full, pitch, roll, warps):
    ship_p, sim_p = _regrouped(str(tmp_path), counts, (1, 2), state0=_edge_state(pitch, roll, full))
    ship, sim = load_model(ship_p, sim_p)
    steps, samples = 12, [4, 12]
    times = [k * sim["dt"] for k in samples]
    en, t_on = np.array(sim["en"], dtype=np.uint8), np.array(sim["tOn"], dtype=np.float64)
    area = np.asarray(sim["area"], dtype=np.float64) * np.linspace(0.9, 1.2, len(sim["ca"]))
    trim_t, heave_t = np.zeros(2), np.zeros(2)
    Jh, gh, eh = adjoint_host_gradient(ship, sim, en, area, t_on, steps, samples, trim_t, heave_t)
    runs = {}
    for budget, every in ((0, 256), (1, 5)):
        with ssb.Adjoint(ship_p, sim_p, count=1, t_max=steps * sim["dt"], checkpoint_every=every, team_warps=warps, tape_budget=budget) as a:
            a.set_connection_areas(0, np.arange(area.size), area[None, :])
            a.set_objective(times, trim_t, heave_t)
            J, g, st, err, _ = a.run()
            runs[every] = J[0], g[0], st[0], err[0], a.recomputed_steps()[0]
    # 12 steps of records fit the smallest ring of 256 steps, not that of 5
    assert runs[256][4] == 0 and runs[5][4] > 0
    for every, (J, g, st, err, _) in runs.items():
        assert (J, st, err) == (Jh, steps, eh), every
    np.testing.assert_array_equal(runs[5][1], runs[256][1])
    if eh == 0:
        np.testing.assert_allclose(runs[256][1], gh, rtol=1e-9, atol=1e-12 * np.max(np.abs(gh)))
    else:  # a branch without an adjoint (an overflow passed down a group), reported alike
        assert full and counts != (1,)
