"""Terrain, mesh and compound queries dealt over a warp, against the oracle:
one column, triangle or part up to more than a warp has lanes, flat terrain
and a flat mesh (every query the same distance: the first must win), fast
movers (casts), and so many compound pairs that they go a thread to a pair.
Discovery and the casts decide integers from these distances, so pair sets,
contact IDs and poses must be identical (error 0), as they are for the
reference's sequential loops."""
import numpy as np
import pytest

from ornis_gb300 import abi, scenes
from ornis_gb300.avbd import AvbdWorld

import oracle_api as O
import parity as P
from test_oracle_shapes_ext import ext_body

pytestmark = pytest.mark.gpu


def ground(kind, cell, flat, rng):
    n = 24
    if kind == "terrain":
        h = np.full((n, n), 0.25) if flat else rng.uniform(0.0, 0.4, (n, n))
        return ("add_heightfield", h, cell)
    xz = (np.arange(n) - n / 2) * cell
    y = np.zeros((n, n)) if flat else rng.uniform(0.0, 0.4, (n, n))
    verts = np.array([[xz[i], y[i, k], xz[k]] for i in range(n) for k in range(n)], np.float32)
    tris = [t for i in range(n - 1) for k in range(n - 1)
            for t in ((i * n + k, i * n + k + 1, (i + 1) * n + k), (i * n + k + 1, (i + 1) * n + k + 1, (i + 1) * n + k))]
    return ("add_trimesh", verts, tris)


def parts():
    S = abi.shape_part
    return [[S(abi.SHAPE_SPHERE, [0.3])],
            [S(abi.SHAPE_BOX, [0.3, 0.1, 0.1]), S(abi.SHAPE_CAPSULE, [0.1, 0.2], position=(0.2, 0.2, 0.0))],
            [S(abi.SHAPE_SPHERE, [0.08], position=(0.25 * (k % 3 - 1), 0.2 * (k // 3 % 3 - 1), 0.2 * (k // 9 - 2)))
             for k in range(40)]]


def pair_of(first, recs, params):
    o, g = O.OracleWorld(params, mode=O.COLOURED), AvbdWorld(params)
    if first:
        assert getattr(o, first[0])(*first[1:]) == (0, getattr(g, first[0])(*first[1:]))
    for p in parts():
        a = o.add_compound(p)
        assert (a[1] if isinstance(a, tuple) else a) == g.add_compound(p)
    bodies = O.bodies_to_array(recs)
    o.add_bodies(bodies)
    g.add_bodies(bodies)
    return o, g


def run(o, g, params, steps):
    pairs = 0
    for _ in range(steps):
        so, sg = P.step_from_oracle_state(o, g)
        assert max(P.compare_states(so, sg, params.step_dt, o, g)) == 0.0
        pairs = max(pairs, len(so["pairs"]))
    return pairs


@pytest.mark.parametrize("kind", ["terrain", "mesh"])
@pytest.mark.parametrize("cell,flat,speed", [(4.0, False, 0.0), (0.5, False, 0.0), (0.25, True, 0.0), (0.2, False, 0.0),
                                             (0.4, False, 50.0)])
def test_bodies_on_ground(kind, cell, flat, speed):
    """Boxes, spheres and compounds of one, two and forty parts; windows of one cell to more than 64."""
    rng = np.random.default_rng(5)
    base = O.body_new(abi.SHAPE_BOX, [1, 1, 1], [0, 0, 0], 0.0)
    base.shape = abi.SHAPE_HEIGHTFIELD if kind == "terrain" else abi.SHAPE_TRIMESH
    base.shape_params[:] = [0.0, 0.0, 0.0]
    recs = [base]
    reach = 10.0 * cell
    for i in range(10):
        pos = [rng.uniform(-reach, reach) * 0.6, 0.9 + 0.1 * i, rng.uniform(-reach, reach) * 0.6]
        k = i % 5
        if k < 3:
            b = ext_body(abi.SHAPE_COMPOUND, k, pos, 1.0, (0.1, 0.1, 0.1))
        elif k == 3:
            b = O.body_new(abi.SHAPE_BOX, [0.7, 0.3, 0.8], pos, 1.0)
        else:
            b = O.body_new(abi.SHAPE_SPHERE, [0.4], pos, 1.0)
        b.orientation[:] = [float(x) for x in scenes.random_quats(rng, 1)[0]]
        if speed:
            b.position[1] += 1.0
            b.velocity[:] = [5.0, -speed, 0.0]
        recs.append(b)
    params = abi.default_params()
    o, g = pair_of(ground(kind, cell, flat, rng), recs, params)
    assert run(o, g, params, 12) > 0


@pytest.mark.parametrize("n", [5, 10])
def test_many_compound_pairs(n):
    """n x n x n compounds in reach of their neighbours: 300 pairs by warps, 2,700 by threads."""
    rng = np.random.default_rng(6)
    recs = []
    for i in range(n):
        for j in range(n):
            for k in range(n):
                b = ext_body(abi.SHAPE_COMPOUND, 0, [0.61 * i, 0.61 * j, 0.61 * k], 1.0, (0.1, 0.1, 0.1))
                if (i + j + k) % 2:
                    b = O.body_new(abi.SHAPE_SPHERE, [0.3], [0.61 * i, 0.61 * j, 0.61 * k], 1.0)
                b.velocity[:] = [float(x) for x in rng.normal(size=3) * 0.3]
                recs.append(b)
    params = abi.default_params(gravity=(0.0, 0.0, 0.0))
    o, g = pair_of(None, recs, params)
    assert run(o, g, params, 3) >= 3 * n * n * (n - 1) - n
