"""Box-box distances taken by a warp, against the oracle: pairs at random
poses, axis-aligned ones (zero cross products, coincident features: the lowest
feature number must win its ties), faces, edges and corners touching and
overlapping; swept casts of fast boxes.  Discovery and the casts decide
integers from these distances, so pair sets, contact IDs and poses must be
identical (error 0), as they are for the reference's sequential loops."""
import numpy as np
import pytest

from ornis_gb300 import abi, scenes

import parity as P

pytestmark = pytest.mark.gpu


def grid_of_pairs(mode, n=40, seed=3):
    """n pairs of boxes, 6 m apart, the second box near, touching or inside the first."""
    rng = np.random.default_rng(seed)
    half = rng.uniform(0.3, 0.7, (2 * n, 3))
    pos = np.zeros((2 * n, 3))
    i = np.arange(n)
    pos[0::2, 0], pos[0::2, 2] = (i % 8) * 6.0, (i // 8) * 6.0
    pos[0::2, 1] = 5.0
    q = scenes.random_quats(rng, 2 * n)
    if mode == "aligned":
        q[:] = [0, 0, 0, 1]
        half[:] = 0.5
        off = rng.choice([-1.0, -0.5, 0.0, 0.5, 1.0], (n, 3))
        off[np.all(off == 0, axis=1)] = [0, 1, 0]
    else:
        off = rng.normal(size=(n, 3))
        off *= (rng.uniform(0.5, 1.6, n) / np.linalg.norm(off, axis=1))[:, None]
    pos[1::2] = pos[0::2] + off
    b = scenes.make_bodies([abi.SHAPE_BOX] * (2 * n), half, pos, np.ones(2 * n), q)
    if mode == "swept":
        pos[1::2] = pos[0::2] + rng.normal(size=(n, 3)) * [3.0, 0.2, 0.2] + [4.0, 0, 0]
        b["position"] = pos
        b["velocity"][1::2] = [-60.0, 0.0, 0.0] + rng.normal(size=(n, 3)) * 5.0
    return b


@pytest.mark.parametrize("mode", ["random", "aligned", "swept"])
def test_box_pairs(mode):
    bodies, params = grid_of_pairs(mode), abi.default_params()
    o, g = P.make_pair(bodies, params)
    pairs = 0
    for _ in range(8):
        so, sg = P.step_from_oracle_state(o, g)
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0
        pairs = max(pairs, len(so["pairs"]))
    assert pairs > 10
