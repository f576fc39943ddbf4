"""The bound on the swept casts' dependency rounds, and what goes with it.

A fast body casts after the earlier fast bodies among its candidates have been
clamped.  The device settles these in eight rounds; a body still waiting is
clamped by its last cast and counted (AvbdCounters.timeouts), where the
reference walks every body in order.  Ten bodies at 40 m/s in one cluster above
terrain are such a chain: a step may differ from the oracle's only if it was
counted, and steps that are not counted are identical (error 0)."""
import numpy as np
import pytest

from ornis_gb300 import abi, scenes

import oracle_api as O
import parity as P
from test_gpu_wide_pairs import ground, pair_of
from test_oracle_shapes_ext import ext_body

pytestmark = pytest.mark.gpu


def cluster(rng, n, speed, reach):
    base = O.body_new(abi.SHAPE_BOX, [1, 1, 1], [0, 0, 0], 0.0)
    base.shape = abi.SHAPE_HEIGHTFIELD
    base.shape_params[:] = [0.0, 0.0, 0.0]
    recs = [base]
    for i in range(n):
        pos = [rng.uniform(-reach, reach) * 0.6, 1.9 + 0.1 * i, rng.uniform(-reach, reach) * 0.6]
        k = i % 5
        if k < 3:
            b = ext_body(abi.SHAPE_COMPOUND, k, pos, 1.0, (0.1, 0.1, 0.1))
        elif k == 3:
            b = O.body_new(abi.SHAPE_BOX, [0.7, 0.3, 0.8], pos, 1.0)
        else:
            b = O.body_new(abi.SHAPE_SPHERE, [0.4], pos, 1.0)
        b.orientation[:] = [float(x) for x in scenes.random_quats(rng, 1)[0]]
        b.velocity[:] = [5.0, -speed, 0.0]
        recs.append(b)
    return recs


@pytest.mark.parametrize("n,chained", [(7, False), (10, True)])
def test_only_counted_steps_differ(n, chained):
    rng = np.random.default_rng(5)
    hf = ground("terrain", 0.25, True, rng)
    params = abi.default_params()
    o, g = pair_of(hf, cluster(rng, n, 40.0, 2.5), params)
    counted = 0
    for _ in range(12):
        before = g.counters().timeouts
        so, sg = P.step_from_oracle_state(o, g)
        if g.counters().timeouts != before:
            counted += 1
            continue
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0
    assert (counted > 0) == chained and counted < 12 and g.counters().ccd_hits > 0
