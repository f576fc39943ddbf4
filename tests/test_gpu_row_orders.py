"""Both orders in which a body's rows are summed (lanes 1: row by row; lanes 0 and
-1: pair by pair), per step from identical state against the oracle in the same
order: batched scenes, ragdolls, a body with 226 pairs, a scene above 2048 bodies.
The oracle is the independent implementation; lanes 0 and -1 are one code
path and only agree with each other by construction."""
import numpy as np
import pytest

from ornis_gb300 import abi, scenes
from ornis_gb300.avbd import AvbdWorld

import oracle_api as O
import parity as P

pytestmark = pytest.mark.gpu

ORDERS = [(1, False), (0, True), (abi.PRIMAL_SCENES, True)]


def check(bodies, params, lanes, split, steps, joints=(), warm=0, nsub=1):
    """Warm the world up on the device, then step both from the oracle's state."""
    o, g = P.make_pair(bodies, params, joints)
    o.split_sums(split)
    g.set_tuning(lanes, 128)
    if warm:
        w = AvbdWorld(params, bodies=bodies)
        for j in joints:
            w.add_joint(j)
        w.set_tuning(lanes, 128)
        w.step_graph(warm)
        o.import_state(w.export_state())
        w.close()
    pairs = 0
    for _ in range(steps):
        so, sg = P.step_from_oracle_state(o, g, nsub)
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0
        pairs = max(pairs, len(so["pairs"]))
    return pairs


@pytest.mark.parametrize("lanes,split", ORDERS)
@pytest.mark.parametrize("n", [30, 250, 600])
def test_bin_scenes(lanes, split, n):
    bodies = scenes.bin_scene(np.random.default_rng([21, n]), n)
    params, nsub = scenes.params_for("batched_4096")
    assert check(bodies, params, lanes, split, 6, warm=600, nsub=nsub) > n // 2


@pytest.mark.parametrize("lanes,split", ORDERS)
def test_ragdolls(lanes, split):
    bodies, offs, joints = scenes.ragdolls((5,), seed=6)
    params, nsub = scenes.params_for("ragdoll_8192")
    assert check(bodies, params, lanes, split, 6, joints, warm=60, nsub=nsub) > 0


@pytest.mark.parametrize("lanes,split", ORDERS)
def test_body_with_226_pairs(lanes, split):
    g = (np.arange(15) - 7) * 0.42
    xs, zs = np.meshgrid(g, g)
    n = xs.size
    bodies = np.concatenate([
        scenes.halfspace([0, 0, 0], [0, 1, 0]),
        scenes.make_bodies([abi.SHAPE_SPHERE] * n, [[0.2, 0, 0]] * n,
                           np.stack([xs.ravel(), np.full(n, 0.2), zs.ravel()], 1), [0.1] * n),
        scenes.make_bodies([abi.SHAPE_BOX], [[3.4, 0.1, 3.4]], [[0.0, 0.5, 0.0]], [20.0])])
    params = abi.default_params(step_dt=1.0 / 120.0, iterations=8)
    assert check(bodies, params, lanes, split, 6, warm=30) >= 2 * n


@pytest.mark.parametrize("lanes,split", ORDERS)
def test_scene_above_2048_bodies(lanes, split):
    bodies = scenes.bin_scene(np.random.default_rng([5, 5]), 2100)
    params, nsub = scenes.params_for("batched_4096")
    assert check(bodies, params, lanes, split, 2, warm=900, nsub=nsub) > 1000
