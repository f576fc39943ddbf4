"""The work that programs have this library do, as a list of cases to time.

A case is one control pass of a program: it writes its body records (new
poses, velocities, drives), advances the world by a few steps and reads the
bodies back, through AvbdWorld; the stateless entry point and the
differentiable rollout are called as their users call them.  Every pass of a
state starts from the same records, so a state can be run any number of
times; the contacts' warm state stays with the world from pass to pass, as it
does for a program that corrects its bodies.

Sizes, steps and iteration counts are those of the repository's workloads
(scenes.py, bench.py), scaled where a whole workload takes longer than a
pass should, and the sizes in between.
"""
import math

import numpy as np

from ornis_gb300 import abi, scenes
from ornis_gb300.avbd import AvbdWorld, Rollout, scene_step_static

F = np.float32


def listed():
    return [
        # a call of the allocation-free entry point: one small scene, host records in and out
        dict(name="static_40", kind="static", bodies=40, steps=2),
        # a small game level stepped through step(dt): where launches count
        dict(name="level_12", kind="level", bodies=12, steps=1, lanes=1),
        # the 210-cube pyramid (20 rows), one step a call
        dict(name="pyramid_210", kind="pyramid", rows=20, steps=1, lanes=1),
        # sprung, driven wheels under 24 chassis among loose bodies: the joint kinds beyond ball and hinge
        dict(name="vehicles_24", kind="vehicles", bodies=24, steps=2, lanes=1),
        # cylinders, cones, hulls, rounded shapes and compounds over a terrain and a mesh
        dict(name="shapes_310", kind="shapes", bodies=310, steps=2, lanes=1),
        # one heap of 1500 boxes, spheres and capsules in a bin, default launch shape
        dict(name="heap_1500", kind="heap", scenes=1, lo=1500, hi=1500, steps=4, lanes=1),
        # 96 environments of a learner, the per-scene solve
        dict(name="envs_96", kind="heap", scenes=96, lo=8, hi=400, steps=4, lanes=-1),
        # the batched workload's piles (body counts log-uniform in 8..1024), the split primal its tuner takes
        dict(name="piles_1536", kind="heap", scenes=1536, lo=8, hi=1024, steps=3, lanes=0),
        # the batched workload while bodies pour in (swept bodies), contact events drained
        dict(name="pour_700", kind="pour", scenes=700, lo=8, hi=1024, steps=4, lanes=0),
        # the large single scene: 100,000 bodies on a plane
        dict(name="plain_100k", kind="field", bodies=100000, steps=3, lanes=0),
        # articulated: two scenes of ragdolls on the ground
        dict(name="ragdolls_1200", kind="ragdolls", bodies=1200, steps=3, lanes=0),
        # the differentiable batch: towers hit by a ball, forward and gradient
        dict(name="towers_grad_96", kind="towers_grad", scenes=96, steps=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["static", "level", "pyramid", "vehicles", "shapes", "heap", "heap", "heap", "pour", "field",
                       "ragdolls", "towers_grad"])
    if kind == "static":
        return dict(kind=kind, bodies=rng.randint(5, 120), steps=rng.randint(1, 4))
    if kind == "level":
        return dict(kind=kind, bodies=rng.randint(5, 160), steps=rng.randint(1, 4), lanes=rng.choice([1, 1, 0, -1]))
    if kind == "pyramid":
        return dict(kind=kind, rows=rng.randint(5, 40), steps=rng.randint(1, 4), lanes=rng.choice([1, 1, 0, -1]))
    if kind == "vehicles":
        return dict(kind=kind, bodies=_log_int(rng, 2, 150), steps=rng.randint(1, 4), lanes=rng.choice([1, 1, 0]))
    if kind == "shapes":
        return dict(kind=kind, bodies=_log_int(rng, 30, 600), steps=rng.randint(1, 3), lanes=rng.choice([1, 1, 0]))
    if kind == "heap":
        if rng.random() < 0.4:
            n = _log_int(rng, 300, 6000)
            return dict(kind=kind, scenes=1, lo=n, hi=n, steps=rng.randint(1, 4), lanes=rng.choice([1, 0]))
        lo = rng.randint(4, 40)
        return dict(kind=kind, scenes=_log_int(rng, 16, 1400), lo=lo, hi=rng.randint(lo, 1000), steps=rng.randint(1, 3),
                    lanes=rng.choice([1, 0, 0, -1]))
    if kind == "pour":
        lo = rng.randint(4, 40)
        return dict(kind=kind, scenes=_log_int(rng, 16, 700), lo=lo, hi=rng.randint(lo, 1000), steps=rng.randint(1, 4),
                    lanes=rng.choice([1, 0, -1]))
    if kind == "field":
        return dict(kind=kind, bodies=_log_int(rng, 3000, 95000), steps=rng.randint(1, 3), lanes=rng.choice([1, 0, 0]))
    if kind == "ragdolls":
        return dict(kind=kind, bodies=_log_int(rng, 8, 1200), steps=rng.randint(1, 3), lanes=rng.choice([1, 0, 0]))
    return dict(kind=kind, scenes=_log_int(rng, 4, 96), steps=rng.randint(4, 12))


# ---- scenes --------------------------------------------------------------------------
def _mixed(rng, n, capsules, big=0.5):
    """n records: boxes, spheres (and capsules) of density 1 and friction U[0.3, 0.8]; no box half-extent or
    radius above `big`, so that a lattice of pitch 3.5 big holds them without overlap."""
    u = rng.random(n)
    kind = np.where(u < 0.6, abi.SHAPE_BOX, abi.SHAPE_SPHERE)
    if capsules:
        kind = np.where(u > 0.9, abi.SHAPE_CAPSULE, kind)
    params = np.zeros((n, 3))
    box, sph, cap = (kind == k for k in (abi.SHAPE_BOX, abi.SHAPE_SPHERE, abi.SHAPE_CAPSULE))
    params[box] = rng.uniform(0.4 * big, big, size=(box.sum(), 3))
    params[sph, 0] = rng.uniform(0.4 * big, big, size=sph.sum())
    params[cap, 0] = 0.4 * big
    params[cap, 1] = rng.uniform(0.3 * big, 1.1 * big, size=cap.sum())
    vol = np.where(box, 8 * params.prod(axis=1), 4.0 / 3.0 * math.pi * params[:, 0] ** 3)
    vol[cap] += math.pi * params[cap, 0] ** 2 * 2 * params[cap, 1]
    return scenes.make_bodies(kind, params, np.zeros((n, 3)), vol, scenes.random_quats(rng, n),
                              rng.uniform(0.3, 0.8, n))


def _bins(rng, nscenes, lo, hi, capsules=False):
    """Scenes of a 20 x 20 bin (5 half-spaces) and log-uniform counts of bodies on a jittered lattice just
    above each other.  Returns (records, scene offsets, mask of the bodies)."""
    half, pitch = 10.0, 1.75
    sizes = np.random.default_rng([nscenes, lo, hi])  # a case's scene sizes are its own, whatever the seed
    counts = np.floor(np.exp(sizes.uniform(math.log(lo), math.log(hi + 1), size=nscenes))).astype(np.int64)
    counts = np.clip(counts, lo, hi)
    planes = np.concatenate([scenes.halfspace(p, n) for p, n in (
        ([0, 0, 0], [0, 1, 0]), ([-half, 0, 0], [1, 0, 0]), ([half, 0, 0], [-1, 0, 0]),
        ([0, 0, -half], [0, 0, 1]), ([0, 0, half], [0, 0, -1]))])
    bodies = _mixed(rng, int(counts.sum()), capsules)
    idx = np.arange(len(bodies)) - np.repeat(np.concatenate([[0], np.cumsum(counts)[:-1]]), counts)
    # a small scene fills the middle of its bin: no wider than needed for three layers
    cols = np.clip(np.ceil(np.sqrt(counts / 3.0)), 2, 11).astype(np.int64)
    cols = np.repeat(cols, counts)
    layer, cell = idx // (cols * cols), idx % (cols * cols)
    off = -(cols - 1) * pitch / 2.0
    pos = np.stack([off + (cell % cols) * pitch, 0.95 + layer * pitch, off + (cell // cols) * pitch], axis=1)
    bodies["position"] = (pos + rng.uniform(-0.05, 0.05, size=pos.shape)).astype(F)
    offs = np.concatenate([[0], np.cumsum(counts + 5)]).astype(np.uint32)
    recs = np.empty(int(offs[-1]), dtype=abi.BODY_DTYPE)
    mask = np.ones(len(recs), dtype=bool)
    for k in range(5):
        mask[offs[:-1] + k] = False
        recs[offs[:-1] + k] = planes[k]
    recs[mask] = bodies
    return recs, offs, mask


def _level(rng, n):
    """A floor, two stacks and falling bodies, and a driven hinge: records and joints."""
    ground = scenes.halfspace([0, 0, 0], [0, 1, 0])
    post = scenes.make_bodies([abi.SHAPE_BOX], [[0.2, 0.2, 0.2]], [[-3, 3, 0]], [0.0])
    arm = scenes.make_bodies([abi.SHAPE_BOX], [[0.1, 0.6, 0.1]], [[-3, 2.2, 0]], [1.0])
    m = max(1, n - 3)
    loose = _mixed(rng, m, True)
    i = np.arange(m)
    loose["position"] = np.stack([(i % 8) * 1.8, 0.9 + 1.2 * (i // 8), rng.uniform(-0.3, 0.3, m)], axis=1).astype(F)
    loose["velocity"] = rng.uniform(-1, 1, (m, 3)).astype(F)
    joints = [abi.joint_desc(abi.JOINT_REVOLUTE, 1, 2, [0, 0, 0], [0, 0.8, 0], [0, 0, 1], [0, 0, 1],
                             motor=(3.0, 20.0))]
    return np.concatenate([ground, post, arm, loose]), joints


def _vehicles(rng, n):
    """n chassis on four sprung, driven wheels each, and a loose box or sphere beside each."""
    recs, joints = [scenes.halfspace([0, 0, 0], [0, 1, 0])], []
    side = int(math.ceil(math.sqrt(n)))
    base = 1
    for k in range(n):
        at = np.array([(k % side) * 5.0, 1.0, (k // side) * 4.0])
        corners = np.array([[x, -0.5, z] for x in (-0.9, 0.9) for z in (-0.7, 0.7)])
        kinds = [abi.SHAPE_BOX] + [abi.SHAPE_SPHERE] * 4
        params = [[1.1, 0.2, 0.5]] + [[0.35, 0, 0]] * 4
        recs.append(scenes.make_bodies(kinds, params, np.concatenate([[at], at + corners]), [20.0, 2.0, 2.0, 2.0, 2.0]))
        for c in range(4):
            joints.append(abi.joint_desc(abi.JOINT_WHEEL, base, base + 1 + c, corners[c], [0, 0, 0], (0, 1, 0), (0, 1, 0),
                                         motor=(float(rng.uniform(2, 8)), 15.0),
                                         wheel=((0, 0, 1), (0, 0, 1), 3.0, 0.7)))
        base += 5
    loose = _mixed(rng, n, False)
    i = np.arange(n)
    loose["position"] = np.stack([(i % side) * 5.0 + 2.0, np.full(n, 0.9), (i // side) * 4.0], axis=1).astype(F)
    loose["velocity"] = rng.uniform(-2, 2, (n, 3)).astype(F)
    return np.concatenate(recs + [loose]), joints


_CUBE_FACES = [(0, 1, 3), (0, 3, 2), (4, 6, 7), (4, 7, 5), (0, 4, 5), (0, 5, 1), (2, 3, 7), (2, 7, 6), (0, 2, 6), (0, 6, 4),
               (1, 5, 7), (1, 7, 3)]


def _shapes(world, rng, n):
    """Every convex shape, rounded and compound ones over a rolling terrain and a mesh slab: records (the shape
    tables go into the world first)."""
    r = 1.0 / math.sqrt(2.0)
    tet = 0.5 * np.array([[1, 0, -r], [-1, 0, -r], [0, 1, r], [0, -1, r]])
    cube = np.array([[x, y, z] for x in (-0.4, 0.4) for y in (-0.3, 0.3) for z in (-0.5, 0.5)])
    ui = (0.1, 0.1, 0.1)
    hulls = [world.add_hull(tet, [(0, 2, 1), (0, 1, 3), (0, 3, 2), (1, 2, 3)], ui), world.add_hull(cube, _CUBE_FACES, ui)]
    rounds = [world.add_round(abi.shape_part(abi.SHAPE_BOX, [0.3, 0.25, 0.35], 0.08), ui),
              world.add_round(abi.shape_part(abi.SHAPE_CYLINDER, [0.3, 0.25], 0.05), ui)]
    comps = [world.add_compound([abi.shape_part(abi.SHAPE_BOX, [0.5, 0.12, 0.12]),
                                 abi.shape_part(abi.SHAPE_BOX, [0.12, 0.35, 0.12], position=(0.4, 0.45, 0))], ui)]
    side = int(math.ceil(math.sqrt(n / 2.0)))
    rows = side + 6
    h = 0.25 * np.sin(0.7 * np.arange(rows))[:, None] * np.cos(0.6 * np.arange(rows))[None, :]
    hf = world.add_heightfield(h + rng.uniform(-0.03, 0.03, h.shape), 1.5)
    slab = [[-4, 0, -4], [4, 0, -4], [4, 0.4, 4], [-4, 0.4, 4]]
    mesh = world.add_trimesh(slab, [(0, 2, 1), (0, 3, 2)])
    kinds = [(abi.SHAPE_CYLINDER, [0.3, 0.35, 0]), (abi.SHAPE_CONE, [0.35, 0.3, 0]), (abi.SHAPE_HULL, [hulls[0], 0, 0]),
             (abi.SHAPE_HULL, [hulls[1], 0, 0]), (abi.SHAPE_BOX, [0.3, 0.25, 0.35]), (abi.SHAPE_SPHERE, [0.3, 0, 0]),
             (abi.SHAPE_CAPSULE, [0.2, 0.3, 0])]
    ext = [(abi.SHAPE_ROUND, rounds[0]), (abi.SHAPE_ROUND, rounds[1]), (abi.SHAPE_COMPOUND, comps[0])]
    shape, params = np.zeros(n, dtype=np.uint32), np.zeros((n, 3))
    for i in range(n):
        k = i % (len(kinds) + len(ext))
        if k < len(kinds):
            shape[i], params[i] = kinds[k]
        else:
            shape[i], params[i, 0] = ext[k - len(kinds)]
    # records as a sphere's, then the shape by its id (the constructors know no tables)
    plain = np.where(shape >= abi.SHAPE_ROUND, abi.SHAPE_SPHERE, shape)
    i = np.arange(n)
    pos = np.stack([(i % side) * 1.5 - 0.75 * side, 0.9 + 1.1 * (i // (side * side)), (i // side % side) * 1.5 - 0.75 * side],
                   axis=1)
    b = scenes.make_bodies(plain, params, pos, np.ones(n), scenes.random_quats(rng, n))
    b["shape"] = shape
    b["inertia"][shape >= abi.SHAPE_HULL] = F(0.1)
    b["rolling_friction"][shape == abi.SHAPE_HULL] = F(0.2)
    b["velocity"] = rng.uniform(-0.5, 0.5, (n, 3)).astype(F)
    ground = scenes.make_bodies([abi.SHAPE_BOX, abi.SHAPE_BOX], [[1, 1, 1]] * 2, [[0, 0, 0], [0.75 * side + 6, 0, 0]],
                                [0.0, 0.0])
    ground["shape"] = [abi.SHAPE_HEIGHTFIELD, abi.SHAPE_TRIMESH]
    ground["shape_params"] = [[hf, 0, 0], [mesh, 0, 0]]
    return np.concatenate([ground, b])


def _field(rng, n):
    """n bodies in three layers on a jittered lattice above a ground plane."""
    b = _mixed(rng, n, True)
    side = int(math.ceil(math.sqrt(n / 3.0)))
    i = np.arange(n)
    layer, cell = i // (side * side), i % (side * side)
    pos = np.stack([(cell % side - side / 2) * 1.4, 0.95 + layer * 1.75, (cell // side - side / 2) * 1.4], axis=1)
    b["position"] = (pos + rng.uniform(-0.1, 0.1, pos.shape)).astype(F)
    return np.concatenate([scenes.halfspace([0, 0, 0], [0, 1, 0]), b])


def _ragdolls(rng, n, seed):
    """Two scenes of n ragdolls in all (a third and two thirds), copies of eight seeded ones on a grid."""
    few, _, fj = scenes.ragdolls(counts=(8,), seed=seed & 0xffff, density=1000.0)
    per = (len(few) - 1) // 8
    jper = len(fj) // 8
    counts = [max(1, n // 3), n - max(1, n // 3)] if n > 1 else [n]
    parts, offs, joints, base = [], [0], [], 0
    for count in counts:
        side = int(math.ceil(math.sqrt(count)))
        pick = rng.integers(0, 8, count)
        parts.append(few[:1])
        for k in range(count):
            r = few[1 + per * pick[k]:1 + per * (pick[k] + 1)].copy()
            lo = (r["position"][:, 1] - r["shape_params"][:, 0] - r["shape_params"][:, 1]).min()
            # the templates' grid places go, this ragdoll's comes; just above the ground
            r["position"] -= np.array([r["position"][0, 0], lo - 0.05, r["position"][0, 2]], dtype=F)
            r["position"] += np.array([(k % side) * 2.5, 0, (k // side) * 2.5], dtype=F)
            first = base + 1 + k * per
            for j in fj[jper * pick[k]:jper * (pick[k] + 1)]:
                d = abi.AvbdJointDesc.from_buffer_copy(j)
                d.body_a = first + (j.body_a - 1) % per
                d.body_b = first + (j.body_b - 1) % per
                joints.append(d)
            parts.append(r)
        base += 1 + count * per
        offs.append(base)
    return np.concatenate(parts), np.asarray(offs, dtype=np.uint32), joints


# ---- passes --------------------------------------------------------------------------
class _State:
    pass


def prepare(case, seed):
    s = _State()
    rng = np.random.default_rng([int(seed) & 0xffffffff, 7])
    s.kind, s.steps = case["kind"], case["steps"]
    kind = s.kind
    s.queue = None
    s.sub, settle = 1, 0
    if kind == "static":
        s.params = abi.default_params()
        s.records = _mixed(rng, case["bodies"] - 1, True)
        i = np.arange(case["bodies"] - 1)
        s.records["position"] = np.stack([(i % 5) * 1.8, 0.85 + 1.0 * (i // 25), (i // 5 % 5) * 1.8], axis=1).astype(F)
        s.records["velocity"] = rng.uniform(-1, 1, (len(i), 3)).astype(F)
        s.records = np.concatenate([scenes.halfspace([0, 0, 0], [0, 1, 0]), s.records])
        return s
    joints, offs = [], None
    if kind == "pyramid":
        # awake throughout, as a learner or a builder's preview runs it
        params = abi.default_params(enable_sleep=0)
        rec = scenes.pyramid_210(seed=int(seed) & 0xffffffff, rows=case["rows"])
        settle = 10
    elif kind == "level":
        params = abi.default_params()
        rec, joints = _level(rng, case["bodies"])
        settle = 16
    elif kind == "vehicles":
        params = abi.default_params()
        rec, joints = _vehicles(rng, case["bodies"])
        settle = 16
    elif kind == "shapes":
        params = abi.default_params()
        w = AvbdWorld(params)
        rec = _shapes(w, rng, case["bodies"])
        w.add_bodies(rec)
        settle = 24
    elif kind in ("heap", "pour"):
        params, s.sub = abi.default_params(step_dt=1.0 / 120.0, iterations=8, enable_sleep=int(kind == "pour")), 2
        rec, offs, mask = _bins(rng, case["scenes"], case["lo"], case["hi"], capsules=case["scenes"] == 1)
        settle = 70 if kind == "heap" else 2
        if kind == "pour":  # bodies that fell from up to 20 m
            s.queue = np.zeros(4 * len(rec), dtype=abi.CONTACT_EVENT_DTYPE)
            v = np.sqrt(2 * 9.81 * rng.uniform(0, 20, int(mask.sum()))).astype(F)
            vel = rec["velocity"].copy()
            vel[mask, 1] = -v
            rec["velocity"] = vel
            pos = rec["position"].copy()
            pos[mask, 1] *= F(1.15)
            rec["position"] = pos
    elif kind == "field":
        params = abi.default_params(enable_sleep=0)
        rec = _field(rng, case["bodies"])
        settle = 50
    elif kind == "ragdolls":
        params, s.sub = abi.default_params(step_dt=1.0 / 120.0, iterations=12), 2
        rec, offs, joints = _ragdolls(rng, case["bodies"], int(seed))
        settle = 30
    elif kind == "towers_grad":
        params = abi.default_params()
        rec, offs, _, tower = scenes.diff_towers(nscenes=case["scenes"], seed=int(seed) & 0xffffffff)
        s.grad = np.zeros((len(rec), 13), dtype=F)
        s.grad[tower, :3] = rng.normal(size=(int(tower.sum()), 3)).astype(F)
    else:
        raise ValueError(kind)
    if kind != "shapes":
        w = AvbdWorld(params, bodies=rec, scene_offsets=offs)
    for d in joints:
        w.add_joint(d)
    if kind == "towers_grad":
        w.set_events(-1)
        s.rollout = Rollout(w, case["steps"], checkpoint_every=6)
    else:
        w.set_tuning(case["lanes"], 128)
        # the program that has run for a while: contacts formed, launch graphs captured
        w.step_graph(max(1, settle * s.sub))
    s.world = w
    s.records = w.bodies() if settle else rec
    s.batch = offs is not None
    return s


def _fields(b):
    return {k: b[k] for k in ("position", "orientation", "velocity", "angular_velocity")}


def run(s):
    if s.kind == "static":
        return _fields(scene_step_static(s.params, s.records, s.steps))
    w = s.world
    w.set_bodies(s.records)
    if s.kind == "towers_grad":
        out = _fields(s.rollout.forward())
        grad, mu = s.rollout.backward(s.grad)
        return dict(out, grad=grad, grad_friction=mu)
    for _ in range(s.steps):
        if s.batch:
            w.step_graph(s.sub)
        else:
            for _ in range(s.sub):
                w.step(w.params.step_dt)
    out = _fields(w.bodies())
    if s.queue is not None:
        ev = w.contact_events()
        s.queue[:len(ev)] = ev[:len(s.queue)]  # the program's own queue
        s.queue[len(ev):] = 0
        out.update({"event_" + k: s.queue[k] for k in ("body_a", "body_b", "kind", "point", "normal")})
    c = w.counters()
    out["pairs"], out["points"] = int(c.pairs), int(c.points)
    return out


# ---- what a pass cannot do without -----------------------------------------------------
def _size(case):
    """(bodies, contact points, joints, substeps, iterations) of a pass, from the case alone."""
    kind, n = case["kind"], case.get("bodies", 0)
    if kind in ("static", "level", "shapes"):
        return n, 3 * n, 1, case["steps"], 10
    if kind == "pyramid":
        n = case["rows"] * (case["rows"] + 1) // 2
        return n, 8 * n, 0, case["steps"], 10
    if kind == "vehicles":
        return 6 * n, 5 * n, 4 * n, case["steps"], 10
    if kind in ("heap", "pour"):
        lo, hi = case["lo"], case["hi"]
        mean = (hi + 1 - lo) / math.log((hi + 1) / lo)  # of a log-uniform count
        n = max(1, int(case["scenes"] * mean))
        return n, (6 if kind == "heap" else 2) * n, 0, 2 * case["steps"], 8
    if kind == "field":
        return n, 5 * n, 0, case["steps"], 10
    if kind == "ragdolls":
        return 15 * n, 8 * n, 14 * n, 2 * case["steps"], 12
    n = 33 * case["scenes"]  # towers: forward, the recomputed forward and the reverse, about two forwards' work
    return n, 8 * n, 0, 4 * case["steps"], 10


def work(case):
    """Bytes: the records in and out, and in each substep the state that outlives it, read and written once
    (336 B a body, 84 B a contact point, 160 B a joint).  Operations: a point's three rows for both of its
    bodies and its dual (about 700), a body's 6 x 6 solve and pose update (about 500), a joint's rows (about
    1200), each iteration, and the narrowphase (about 2500 a body) each substep."""
    n, points, joints, subs, iters = _size(case)
    return {"bytes": 2.0 * 136 * n + subs * 2.0 * (336 * n + 84 * points + 160 * joints),
            "flops": float(subs) * (iters * (700 * points + 500 * n + 1200 * joints) + 2500 * n)}


def exact(case, seed):
    """No value: the step is a sequence of decisions (contact sets, clamps, the sweep's colours) taken on 32-bit
    values, and a 64-bit run takes others; what a step gives has no 64-bit value short of a second engine."""
    return None
