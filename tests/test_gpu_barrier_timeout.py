"""A grid barrier that gives up (its poll limit set to none, so that a block
that arrives before the others returns at once): the call reports
AVBD_ERR_TIMEOUT, no later kernel of the substep runs on what was left
unfinished, and the world takes no steps and gives no snapshot until a whole
state is imported; from that state it then steps as a new world does."""
import ctypes as C

import numpy as np
import pytest

from ornis_gb300 import abi, scenes
from ornis_gb300.avbd import AvbdError, AvbdWorld, Rollout, lib

from test_gpu_tile_engine import pile

pytestmark = pytest.mark.gpu

DEFAULT = 1 << 23


def polls(w, n):
    fn = lib().avbd_test_barrier_polls
    fn.argtypes = [C.c_void_p, C.c_uint32]
    assert fn(w.h, n) == 0


def code(call, *args):
    with pytest.raises(AvbdError) as e:
        call(*args)
    return e.value.code


def falling(n):
    """Bodies fast enough to be swept, none touching."""
    i = np.arange(n)
    b = scenes.make_bodies([abi.SHAPE_SPHERE] * n, [[0.3, 0, 0]] * n,
                           np.stack([(i % 30) * 1.5, 3.0 + 1.5 * (i // 900), (i // 30 % 30) * 1.5], axis=1), np.ones(n))
    b["velocity"][:, 1] = -100.0
    return np.concatenate([scenes.halfspace([0, 0, 0], [0, 1, 0]), b])


WHERE = {"iterations": (pile(700), 1), "swept casts": (falling(700), 1), "large scene": (pile(2500), 2)}


@pytest.mark.parametrize("where", list(WHERE))
@pytest.mark.parametrize("how", ["step_fixed", "step_graph", "profile"])
def test_give_up_is_reported_and_refuses_steps(where, how):
    bodies, warm = WHERE[where]
    w = AvbdWorld(abi.default_params(), bodies=bodies)
    if where != "swept casts":
        (w.step_graph if how == "step_graph" else w.step_fixed)(warm)
    before = w.export_state()
    counted = w.counters()
    polls(w, 0)
    step = {"step_fixed": lambda: w.step_fixed(3), "step_graph": lambda: w.step_graph(3), "profile": w.profile_substep}[how]
    assert code(step) == abi.AVBD_ERR_TIMEOUT
    c = w.counters()
    assert c.steps == counted.steps and c.timeouts > counted.timeouts
    if where != "iterations":  # what follows the barrier did not move a body
        np.testing.assert_array_equal(w.bodies()["position"], before["bodies"]["position"])
    for again in (step, lambda: w.step(1 / 60), w.snapshot):
        assert code(again) == abi.AVBD_ERR_TIMEOUT
    polls(w, DEFAULT)
    assert code(step) == abi.AVBD_ERR_TIMEOUT
    w.import_state(before)
    fresh = AvbdWorld(abi.default_params(), bodies=bodies)
    fresh.import_state(before)
    for x in (w, fresh):
        x.step_graph(3)
    assert w.bodies().tobytes() == fresh.bodies().tobytes()


def test_give_up_in_a_rollout():
    bodies, offs, _, _ = scenes.diff_towers(nscenes=20)
    w = AvbdWorld(abi.default_params(), bodies=bodies, scene_offsets=offs)
    w.set_events(-1)
    r = Rollout(w, 6, checkpoint_every=3)
    r.forward()
    polls(w, 0)
    g = np.ones((len(bodies), 13), np.float32)
    assert code(r.backward, g) == abi.AVBD_ERR_TIMEOUT
    polls(w, DEFAULT)
    assert code(r.backward, g) == abi.AVBD_ERR_TIMEOUT
    assert code(r.forward) == abi.AVBD_ERR_TIMEOUT
