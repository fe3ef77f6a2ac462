"""Models whose spaces share free surfaces in large groups: the engine picks team sizes whose pass buffers fit, and steps
them like the C restatement."""
import json

import numpy as np
import pytest

import sinksim_b200 as ssb
from _support import Oracle, load_model
from sinksim_b200 import hullgen

pytestmark = pytest.mark.gpu

STEPS = 8


def one_group(out, spec):
    """A generated hull with all its spaces in one group that always shares its surface."""
    ship_p, sim_p = hullgen.write(out, spec=spec)
    sim = json.load(open(sim_p))
    n = len(sim["state0"]["vol"])
    sim["groups"] = dict(sim["groups"], n=1, nodeStart=[0], nodeCount=[n], mode=[1], px=[0.0], py=[0.0], pz=[4.0])
    sim["connections"]["skipGroup"] = [-1] * sim["connections"]["n"]
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
    ship_p, sim_p = one_group(str(tmp_path), spec)
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
