"""The tile engine (every iteration of a substep in one launch) at the sizes
where its work division changes, per step from identical state against the
oracle: one body, a warp's 32 lanes and one more, the last world a cluster's
barrier holds (512 bodies) and the first the grid's does, bodies with more
items than a round's 32, rolling friction (the dual in its own pass), joints
of every tier.  The engine makes the oracle's additions in the oracle's order,
so the exact build must be bit-identical (asserted as error 0); the split
order of lanes 0 equals that of lanes -1 bit for bit."""
import numpy as np
import pytest

from ornis_gb300 import abi, scenes
from ornis_gb300.avbd import AvbdWorld

import parity as P

pytestmark = pytest.mark.gpu


def pile(n, seed=5, rolling=0.0):
    """Half-space plus n - 1 boxes, spheres and capsules resting on one another in tight columns."""
    rng = np.random.default_rng(seed)
    m = n - 1
    kind = rng.choice([abi.SHAPE_BOX, abi.SHAPE_BOX, abi.SHAPE_SPHERE, abi.SHAPE_CAPSULE], m)
    params = np.where((kind == abi.SHAPE_BOX)[:, None], 0.5, np.array([0.5, 0.0, 0.0]))
    params[kind == abi.SHAPE_CAPSULE] = [0.3, 0.25, 0.0]
    side = max(1, int(np.ceil((m / 3.0) ** 0.5)))
    i = np.arange(m)
    pos = np.stack([(i % side) * 1.02, 0.5 + 1.0 * (i // (side * side)), (i // side % side) * 1.02], axis=1)
    pos[:, [0, 2]] += rng.uniform(-0.01, 0.01, (m, 2))
    b = scenes.make_bodies(kind, params, pos, np.ones(m))
    b["rolling_friction"] = rolling
    b["torsion_friction"] = 0.5 * rolling
    return np.concatenate([scenes.halfspace([0, 0, 0], [0, 1, 0]), b])


@pytest.mark.parametrize("n", [2, 33, 34, 129, 512, 513, 700])
def test_pile_sizes(n):
    bodies, params = pile(n), abi.default_params()
    o, g = P.make_pair(bodies, params)
    for _ in range(12):
        so, sg = P.step_from_oracle_state(o, g)
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0


def test_rolling_friction():
    bodies, params = pile(60, rolling=0.2), abi.default_params()
    o, g = P.make_pair(bodies, params)
    for _ in range(12):
        so, sg = P.step_from_oracle_state(o, g)
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0


def test_many_contacts_on_one_body():
    """A slab under 60 cubes (240 points: eight rounds of one body) with a joint of every row tier."""
    rng = np.random.default_rng(2)
    slab = scenes.make_bodies([abi.SHAPE_BOX], [[6.0, 0.25, 6.0]], [[0, 0.26, 0]], [50.0])
    i = np.arange(60)
    cubes = scenes.make_bodies([abi.SHAPE_BOX] * 60, np.full((60, 3), 0.4),
                               np.stack([(i % 8) * 1.2 - 4.2, np.full(60, 0.91), (i // 8) * 1.2 - 4.2], axis=1), np.ones(60))
    cubes["velocity"] = rng.uniform(-0.1, 0.1, (60, 3)).astype(np.float32)
    bodies = np.concatenate([scenes.halfspace([0, 0, 0], [0, 1, 0]), slab, cubes])
    axes = [(-0.2, 0.2), "locked", "free", (-0.1, 0.1), "locked", "free"]
    joints = [abi.joint_desc(abi.JOINT_BALL, 1, 2, [-4.2, 0.25, -4.2], [0, -0.4, 0]),
              abi.joint_desc(abi.JOINT_REVOLUTE, 1, 3, [-3.0, 0.25, -4.2], [0, -0.4, 0], (0, 1, 0), (0, 1, 0), (-0.1, 0.1)),
              abi.joint_desc(abi.JOINT_SIXDOF, 1, 4, [-1.8, 0.25, -4.2], [0, -0.4, 0], axes=axes)]
    params = abi.default_params()
    for js in ([], joints[:2], joints):
        o, g = P.make_pair(bodies, params, js)
        for _ in range(10):
            so, sg = P.step_from_oracle_state(o, g)
            assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0


def test_split_order_forms_agree():
    res = []
    for lanes in (0, -1):
        w = AvbdWorld(abi.default_params(), bodies=pile(300))
        w.set_tuning(lanes, 128)
        w.step_graph(30)
        res.append(w.bodies())
    np.testing.assert_array_equal(res[0], res[1])
