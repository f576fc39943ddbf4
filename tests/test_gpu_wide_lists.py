"""The filter, the build and the swept casts of wide pairs (terrain, meshes,
compounds) by threads, by warps and one of each (test_gpu_wide_pairs.py's lists
are all short enough for warps but one kernel's): each form forced on the same
scenes, per step from identical state against the oracle (error 0).  The casts'
list holds box pairs and wide pairs, so that a cast dropped or made twice by
the split between warps and threads would show."""
import numpy as np
import pytest

from ornis_gb300 import abi, scenes

import oracle_api as O
import parity as P
from test_gpu_pair_lists import FORMS, force
from test_gpu_wide_pairs import ground, pair_of
from test_oracle_shapes_ext import ext_body

pytestmark = pytest.mark.gpu


def records(rng, kind, fast, reach):
    """Ground, six compounds, four boxes and two spheres in two clusters, falling."""
    base = O.body_new(abi.SHAPE_BOX, [1, 1, 1], [0, 0, 0], 0.0)
    base.shape = abi.SHAPE_HEIGHTFIELD if kind == "terrain" else abi.SHAPE_TRIMESH
    base.shape_params[:] = [0.0, 0.0, 0.0]
    recs = [base]
    for i in range(12):
        at = -1.0 if i % 2 else 1.0
        pos = [at * 0.4 * reach + rng.uniform(-0.7, 0.7), 0.9 + 0.35 * i, rng.uniform(-0.7, 0.7)]
        if i < 6:
            b = ext_body(abi.SHAPE_COMPOUND, i % 3, pos, 1.0, (0.1, 0.1, 0.1))
        elif i < 10:
            b = O.body_new(abi.SHAPE_BOX, [0.5, 0.2, 0.6], pos, 1.0)
        else:
            b = O.body_new(abi.SHAPE_SPHERE, [0.35], pos, 1.0)
        b.orientation[:] = [float(x) for x in scenes.random_quats(rng, 1)[0]]
        if fast:
            b.velocity[:] = [2.0, -45.0, 0.0]
        recs.append(b)
    return recs


@pytest.mark.parametrize("longest", [2] + FORMS)
@pytest.mark.parametrize("kind", ["terrain", "mesh"])
@pytest.mark.parametrize("fast", [False, True])
def test_forms(kind, fast, longest):
    rng = np.random.default_rng(17)
    recs = records(rng, kind, fast, 4.0)
    params = abi.default_params()
    o, g = pair_of(ground(kind, 0.4, False, rng), recs, params)
    force(g, longest)
    pairs = 0
    for _ in range(12):
        so, sg = P.step_from_oracle_state(o, g)
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0
        pairs = max(pairs, len(so["pairs"]))
    c = g.counters()
    assert pairs >= 4 and (c.ccd_hits > 5) == fast
