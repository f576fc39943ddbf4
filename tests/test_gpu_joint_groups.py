"""Velocity impulses of motors and ropes taken group by group (joints connected
through dynamic bodies), per step from identical state against the oracle,
which walks them joint by joint: separate mechanisms, a chain whose motors
and ropes share bodies, mechanisms that share only a static body, joints added
out of order.  Bit-identical (error 0)."""
import numpy as np
import pytest

from ornis_gb300 import abi, scenes

import parity as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [0, 1])
def test_mechanisms(order):
    box, ball = [0.2, 0.2, 0.2], [0.25, 0.0, 0.0]
    n, kinds, params, pos, mass, joints = 2, [abi.SHAPE_BOX], [box], [[0, 4, 0]], [0.0], []
    ground = scenes.halfspace([0, 0, 0], [0, 1, 0])
    for k in range(7):  # driven wheels on sprung chassis, apart from each other
        x = 3.0 * k - 9.0
        kinds += [abi.SHAPE_BOX, abi.SHAPE_SPHERE, abi.SHAPE_SPHERE]
        params += [[0.8, 0.2, 0.4], ball, ball]
        pos += [[x, 0.9, 3], [x - 0.6, 0.4, 3], [x + 0.6, 0.4, 3]]
        mass += [5.0, 1.0, 1.0]
        for c in (1, 2):
            joints.append(abi.joint_desc(abi.JOINT_WHEEL, n, n + c, [-0.6 if c == 1 else 0.6, -0.5, 0], [0, 0, 0], (0, 1, 0),
                                         (0, 1, 0), motor=(4.0 + k, 10.0), wheel=((0, 0, 1), (0, 0, 1), 3.0, 0.7)))
        n += 3
    for k in range(3):  # ropes and free motors from one static anchor, each with its own chain
        kinds += [abi.SHAPE_SPHERE] * 3
        params += [ball] * 3
        pos += [[0.8 * k, 3.0 - 0.7 * i, 0.1 * k] for i in range(3)]
        mass += [1.0] * 3
        for i in range(3):
            a = 1 if i == 0 else n + i - 1
            joints.append(abi.joint_desc(abi.JOINT_ROPE, a, n + i, [0, 0, 0], [0, 0, 0], max_distance=0.75 + 0.8 * k * (i == 0)))
        joints.append(abi.joint_desc(abi.JOINT_MOTOR, n, n + 2, [0, 0, 0], [0, 0, 0],
                                     drive=((0.3, 0.0, 0.2), (0.0, 1.0, 0.0), 2.0, 0.1, 0.0)))
        n += 3
    if order:
        joints = joints[1::2] + joints[0::2]
    bodies = np.concatenate([ground, scenes.make_bodies(kinds, params, pos, mass)])
    p = abi.default_params()
    o, g = P.make_pair(bodies, p, joints)
    for _ in range(40):
        so, sg = P.step_from_oracle_state(o, g)
        assert max(P.compare_states(so, sg, p.step_dt, o, g)) == 0.0
