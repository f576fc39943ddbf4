"""Swept casts of a small world whose bodies all move fast: bit-identical to
the oracle on either side of the sizes where the launch changes, and as fast at
500 bodies as the launch for a few more is."""
import numpy as np
import pytest

from ornis_gb300 import abi, scenes
from ornis_gb300.avbd import AvbdWorld

import parity as P

pytestmark = pytest.mark.gpu


def burst(n, pitch, speed, seed=1):
    """n tilted boxes on a lattice falling at `speed` (the lattice is scattered by 5 m/s)."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    pos = np.stack([(i % side) * pitch, 1.0 + (i // side % side) * pitch, (i // (side * side)) * pitch], axis=1)
    b = scenes.make_bodies([abi.SHAPE_BOX] * n, rng.uniform(0.15, 0.3, (n, 3)), pos, np.ones(n),
                           scenes.random_quats(rng, n))
    v = rng.normal(size=(n, 3)) * 5.0
    v[:, 1] -= speed
    b["velocity"] = v.astype(np.float32)
    return np.concatenate([scenes.halfspace([0, 0, 0], [0, 1, 0]), b])


@pytest.mark.parametrize("n", [3, 60, 64, 70, 300])
def test_bursts_against_oracle(n):
    bodies, params = burst(n, 3.0, 60.0), abi.default_params()
    o, g = P.make_pair(bodies, params)
    for _ in range(4):
        so, sg = P.step_from_oracle_state(o, g)
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0
    assert g.counters().ccd_hits > 0


def test_time_of_a_burst_of_500():
    """500 bodies against 520: 32 warps had taken all casts of the former, 2.8 times as long."""
    ms = []
    for n in (500, 520):
        rec = burst(n, 0.8, 60.0)
        w = AvbdWorld(abi.default_params(), bodies=rec)
        w.step_graph(2)
        t = []
        for _ in range(6):
            w.set_bodies(rec)
            t.append(w.profile_substep()[0]["ccd"])
        ms.append(np.median(t[1:]))
        w.close()
    print(f"casts of 500 bodies {ms[0]:.2f} ms, of 520 {ms[1]:.2f} ms")
    assert ms[0] < 1.6 * ms[1]
