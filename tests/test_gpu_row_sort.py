"""The cell-row sweep of large scenes away from the origin and beyond the
one-launch sort: the candidate set is the one-axis sweep's (same counters and
bodies bit for bit), and the time does not depend on where the scene lies."""
import numpy as np
import pytest

from ornis_gb300 import abi, scenes
from ornis_gb300.avbd import AvbdWorld

pytestmark = pytest.mark.gpu


def field(n, shift, pitch=1.4, seed=4):
    """n boxes and spheres in one layer above a ground plane, moved `shift` along x."""
    rng = np.random.default_rng(seed)
    kind = np.where(rng.random(n) < 0.5, abi.SHAPE_BOX, abi.SHAPE_SPHERE)
    side = int(np.ceil(np.sqrt(n)))
    i = np.arange(n)
    pos = np.stack([(i % side - side / 2) * pitch, np.full(n, 0.6), (i // side - side / 2) * pitch], axis=1)
    pos[:, [0, 2]] += rng.uniform(-0.15, 0.15, (n, 2))
    b = scenes.make_bodies(kind, np.where((kind == abi.SHAPE_BOX)[:, None], 0.5, [[0.5, 0, 0]]), pos, np.ones(n))
    b["position"][:, 0] += np.float32(shift)
    return np.concatenate([scenes.halfspace([0, 0, 0], [0, 1, 0]), b])


def both_sweeps(bodies, steps):
    counts = []
    out = []
    for rows in (1, 0):
        w = AvbdWorld(abi.default_params(), bodies=bodies)
        w.set_broadphase(0)
        w.set_sweep(rows)
        w.step_fixed(steps)
        c = w.counters()
        counts.append((c.candidates, c.pairs, c.points))
        out.append(w.bodies().tobytes())
        w.close()
    assert counts[0] == counts[1] and counts[0][0] > 0
    assert out[0] == out[1]


@pytest.mark.parametrize("shift", [0.0, 60.0, 300.0, -1e4, 3e3, 1e5])
def test_candidates_away_from_the_origin(shift):
    both_sweeps(field(4000, shift, pitch=1.1), 3)


def test_candidates_beyond_the_one_launch_sort():
    """More bodies than the one-launch sort holds (8 rounds of 256 keys in 304 tiles): the two radix sorts."""
    both_sweeps(field(640000, 2e3), 1)


def test_time_away_from_the_origin():
    """Broadphase of 100,000 bodies 100 km out against the same at the origin.  The work is the same there; a
    sort key of 16 bits of x made it 5 times as long."""
    ms = []
    for shift in (0.0, 1e5):
        w = AvbdWorld(abi.default_params(enable_sleep=0), bodies=field(100000, shift))
        w.step_graph(2)
        ms.append(np.median([w.profile_substep()[0]["broadphase"] for _ in range(9)]))
        w.close()
    print(f"broadphase at the origin {ms[0]:.3f} ms, 100 km out {ms[1]:.3f} ms")
    assert ms[1] < 2.0 * ms[0]
