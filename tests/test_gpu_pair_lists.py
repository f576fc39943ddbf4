"""Discovery and the swept casts by warps and by threads (lists of box pairs and
of wide pairs: terrain, meshes, compounds), each form forced on the same
scenes, per step from identical state against the oracle: pair sets, contact
IDs and poses identical (error 0)."""
import ctypes as C

import numpy as np
import pytest

from ornis_gb300 import abi, scenes
from ornis_gb300.avbd import AvbdWorld, lib

import oracle_api as O
import parity as P

pytestmark = pytest.mark.gpu

# longest list that goes by warps: none, some of a scene's lists, all
FORMS = [0, 30, 0xffffffff]


def force(w, n):
    fn = lib().avbd_test_warp_lists
    fn.argtypes = [C.c_void_p, C.c_uint32]
    assert fn(w.h, n) == 0


def boxes(n, fast):
    """Tilted boxes, thin and cubic, falling on one another in tight columns."""
    rng = np.random.default_rng(11)
    side = int(np.ceil((n / 3.0) ** 0.5))
    i = np.arange(n)
    pos = np.stack([(i % side) * 0.9, 0.5 + 0.8 * (i // (side * side)), (i // side % side) * 0.9], axis=1)
    half = rng.uniform(0.2, 0.5, (n, 3))
    half[::5, 1] = 0.05
    b = scenes.make_bodies([abi.SHAPE_BOX] * n, half, pos, np.ones(n), scenes.random_quats(rng, n))
    if fast:
        b["velocity"][::9, 1] = -60.0
        b["position"][::9, 1] += 4.0
    return np.concatenate([scenes.halfspace([0, 0, 0], [0, 1, 0]), b])


@pytest.mark.parametrize("longest", FORMS)
@pytest.mark.parametrize("n,fast", [(5, False), (33, True), (90, True)])
def test_box_pairs(longest, n, fast):
    bodies, params = boxes(n, fast), abi.default_params()
    o, g = P.make_pair(bodies, params)
    force(g, longest)
    pairs = 0
    for _ in range(10):
        so, sg = P.step_from_oracle_state(o, g)
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0
        pairs = max(pairs, len(so["pairs"]))
    assert pairs >= n // 2 and g.counters().timeouts == 0


def test_forms_agree_on_a_long_list():
    """A list of box pairs beyond four a warp of the launch (38,912): the rule's own choice against threads'."""
    bodies, offs, _ = scenes.batched(300, seed=5, lo=300, hi=1000)
    params, nsub = scenes.params_for("batched_4096")
    out = []
    for longest in (0xffffffff, 0):
        w = AvbdWorld(params, bodies=bodies, scene_offsets=offs)
        force(w, longest)
        w.step_graph(160 * nsub)
        out.append((w.bodies().tobytes(), w.counters().pairs))
        w.close()
    assert out[0] == out[1] and out[0][1] > 100000
