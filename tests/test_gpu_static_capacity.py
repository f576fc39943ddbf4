"""avbd_scene_step_static at the edge of its pair array (2048 candidates) and of
the solver's 64 colours: 64 spheres in one place (2016 contacts, every pair
its own colour step) are stepped as a world steps them; 65 have more pairs
than the array holds: AVBD_ERR_CAPACITY, the output untouched, however many
substeps, and the next call as good as new."""
import ctypes as C

import numpy as np
import pytest

from ornis_gb300 import abi, scenes
from ornis_gb300.avbd import AvbdWorld, lib, scene_step_static

pytestmark = pytest.mark.gpu


def crowd(n):
    rng = np.random.default_rng(3)
    return scenes.make_bodies([abi.SHAPE_SPHERE] * n, [[0.5, 0, 0]] * n, rng.uniform(-0.1, 0.1, (n, 3)), np.ones(n))


def test_crowd_at_and_beyond_capacity():
    params = abi.default_params(gravity=(0.0, 0.0, 0.0))
    for n in (12, 64):
        w = AvbdWorld(params, bodies=crowd(n))
        w.step_fixed(1)
        assert w.counters().colours == n
        got = scene_step_static(params, crowd(n), 1)
        assert np.array_equal(got["position"], w.bodies()["position"])
        w.close()
    good = scene_step_static(params, crowd(12), 3)
    many = crowd(65)
    for substeps in (1, 20):
        out = np.full(65 * abi.BODY_DTYPE.itemsize, 0x5a, np.uint8)
        rc = lib().avbd_scene_step_static(C.byref(params), many.ctypes.data, 65, substeps, out.ctypes.data)
        assert rc == abi.AVBD_ERR_CAPACITY and np.all(out == 0x5a)
    assert scene_step_static(params, crowd(12), 3).tobytes() == good.tobytes()
