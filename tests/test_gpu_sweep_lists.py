"""The small scenes' warp sweep and the large scenes' one-launch colouring
against the oracle, per step from identical state (error 0): scenes around the
sweep's 32-slot stride, a batch of scenes side by side (no pair crosses two
scenes), and one scene taken once as a small and once as a large one (the
colours and candidates must not depend on it)."""
import numpy as np
import pytest

from ornis_gb300 import abi
from ornis_gb300.avbd import AvbdWorld

import parity as P
from test_gpu_tile_engine import pile

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 32, 34, 66, 300])
def test_small_scene(n):
    bodies, params = pile(n, seed=n), abi.default_params()
    o, g = P.make_pair(bodies, params)
    for _ in range(4):
        so, sg = P.step_from_oracle_state(o, g)
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0


def test_batch_equals_each_scene_alone():
    scenes = [pile(n, seed=n) for n in (2, 33, 90, 65, 5)]
    offs = np.concatenate([[0], np.cumsum([len(s) for s in scenes])])
    w = AvbdWorld(abi.default_params(), bodies=np.concatenate(scenes), scene_offsets=offs)
    w.step_graph(25)
    got = w.bodies()
    for k, s in enumerate(scenes):
        a = AvbdWorld(abi.default_params(), bodies=s)
        a.step_graph(25)
        np.testing.assert_array_equal(got[offs[k]:offs[k + 1]], a.bodies())


def test_small_and_large_paths_agree():
    res = []
    for small_max in (2048, 0):
        w = AvbdWorld(abi.default_params(), bodies=pile(900, seed=1))
        w.set_broadphase(small_max)
        w.step_graph(25)
        c = w.counters()
        res.append((w.bodies(), w.colours(), (c.candidates, c.pairs, c.points, c.colours)))
    np.testing.assert_array_equal(res[0][0], res[1][0])
    np.testing.assert_array_equal(res[0][1], res[1][1])
    assert res[0][2] == res[1][2]
