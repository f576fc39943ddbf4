"""Worlds on either side of the sizes where a launch changes its form: the
iterations' barrier (a cluster's up to 400 bodies, a grid's beyond) against the
oracle, and the colours' lists (one block, or a radix sort beyond 16,384
bodies) against the sorted order, whose bodies must be bit-identical."""
import pytest

from ornis_gb300 import abi
from ornis_gb300.avbd import AvbdWorld

import parity as P
from test_gpu_tile_engine import pile

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [399, 400, 401, 416])
def test_cluster_and_grid_barrier(n):
    bodies, params = pile(n, seed=7), abi.default_params()
    o, g = P.make_pair(bodies, params)
    for _ in range(8):
        so, sg = P.step_from_oracle_state(o, g)
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0


@pytest.mark.parametrize("n", [1024, 16384, 16385])
def test_colour_lists(n):
    out = []
    for by_work in (0, 1):  # 1: always the radix sort
        w = AvbdWorld(abi.default_params(), bodies=pile(n, seed=8))
        w.set_work_order(by_work)
        w.step_graph(6)
        out.append((w.bodies().tobytes(), w.counters().colours))
        w.close()
    assert out[0] == out[1] and out[0][1] > 1
