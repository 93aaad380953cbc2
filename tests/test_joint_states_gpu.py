"""Joints of every type in double, where two lanes share a row, against
states recorded from the same engine with one lane a row and one thread
walking the reference's list (tests/golden/joints/record.py), bit for bit:
chains of each type, limited, damped and driven, one damped joint among
undamped ones, the single-joint worlds of test_joints_gpu.py, and joints of a
body with itself."""
import os

import numpy as np
import pytest

from rbps_b200 import abi, scenes
from helpers import GOLDEN
from test_joints_gpu import CASES, I, X, Y, Z, _quat, _world

RECORDED = os.path.join(GOLDEN, "joints", "states.npz")
STEPS = (1, 12)
SOLVES = {"reference": abi.SOLVE_REFERENCE_ORDER, "colored": abi.SOLVE_COLORED}


def chain(n=9, bend=0.0, **kw):
    """n links along x from a static base, each joined to the one before."""
    links = [((0.5 * (k + 1), 0.0, 0.0), _quat(Z, bend * k), 1.0 + 0.1 * k, (0.2, 0.1, 0.1)) for k in range(n)]
    joints = [dict(dict(body_1=k, body_2=k + 1, r_1=(0.25, 0.0, 0.0), r_2=(-0.25, 0.0, 0.0)), **kw) for k in range(n)]
    return links, joints


def jointed_worlds():
    """(name, world) of every case."""
    P, R, F, S = abi.JOINT_PRISMATIC, abi.JOINT_REVOLUTE, abi.JOINT_FIXED, abi.JOINT_SPHERICAL
    hinge = dict(type=R, axis=Z, limit_axis=X)
    cases = dict(CASES)
    cases["chain_revolute"] = chain(**hinge)
    cases["chain_revolute_damped"] = chain(damping=2.0, **hinge)
    cases["chain_revolute_limited"] = chain(limited=1, lower_limit=-0.1, upper_limit=0.05, compliance=1e-4, **hinge)
    cases["chain_revolute_driven"] = chain(actuation=abi.ACTUATION_POSITION, target_position=0.2, compliance=1e-3, **hinge)
    cases["chain_prismatic"] = chain(type=P, axis=Y)
    cases["chain_prismatic_damped"] = chain(type=P, axis=Y, damping=3.0)
    cases["chain_prismatic_limited"] = chain(type=P, axis=Y, limited=1, lower_limit=-0.02, upper_limit=0.01, damping=1.0)
    cases["chain_fixed"] = chain(type=F)
    cases["chain_ball"] = chain(bend=0.2, type=S, axis=X)
    cases["chain_ball_cone"] = chain(bend=0.3, type=S, axis=X, limited=1, upper_limit=0.2, compliance=1e-5)
    links, joints = chain(**hinge)
    joints[4]["damping"] = 2.0
    cases["chain_one_damped"] = (links, joints)
    links, joints = chain(**hinge)
    for k, j in enumerate(joints):
        j.update([dict(), dict(type=F), dict(type=S, axis=X), dict(type=P, axis=Y, damping=1.0)][k % 4])
    cases["chain_mixed"] = (links, joints)
    cases["ring"] = (links, chain(**hinge)[1] + [dict(body_1=1, body_2=8, r_1=(0.0, 0.5, 0.0), r_2=(0.0, 0.5, 0.0), type=S, axis=X)])
    for name, kw in (("fixed", dict(type=F)), ("ball", dict(type=S, axis=X)), ("hinge", hinge), ("prismatic", dict(type=P, axis=Y))):
        cases["self_" + name] = ([((0.0, 1.0, 0.0), _quat(Z, 0.3), 1.0, (0.2, 0.1, 0.1))],
                                 [dict(dict(body_1=1, body_2=1, r_1=(0.1, 0.0, 0.0), r_2=(-0.05, 0.1, 0.0)), **kw)])
    out = []
    for name in sorted(cases):
        spec = _world(*cases[name])
        rng = np.random.default_rng(len(out))
        if name.startswith(("chain", "ring", "self")):
            spec.bodies["linear_velocity"][1:] = rng.uniform(-0.5, 0.5, (len(spec.bodies) - 1, 3))
            spec.bodies["angular_velocity"][1:] = rng.uniform(-0.5, 0.5, (len(spec.bodies) - 1, 3))
        out.append((name, spec))
    return out


def states(rbps, solve):
    """{"<world> <steps> <field>": array} of a batch of all the worlds."""
    worlds = jointed_worlds()
    sc = scenes.Scene("joints", 1.0 / 60.0, 4, 0, [spec for _, spec in worlds])
    b = rbps.Batch.from_scene(sc, abi.PRECISION_FP64, solve)
    b.set_state_check(False)  # some of the single-joint worlds go non-finite, in the reference too
    out, done = {}, 0
    for n in STEPS:
        b.step(n - done)
        done = n
        for w, (name, _) in enumerate(worlds):
            for f, v in b.state(w).items():
                out["%s %d %s" % (name, n, f)] = v
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("solve", sorted(SOLVES))
def test_states_as_recorded(rbps, solve):
    got = states(rbps, SOLVES[solve])
    with np.load(RECORDED) as want:
        names = [k[len(solve) + 1:] for k in want.files if k.startswith(solve + " ")]
        assert sorted(names) == sorted(got)
        for k in names:
            np.testing.assert_array_equal(got[k], want[solve + " " + k], err_msg=k)


def test_recorded_worlds_move():
    """Every chain is finite and none is at rest in the recorded states."""
    with np.load(RECORDED) as want:
        for k in want.files:
            name = k.split()[1]
            if name.startswith(("chain", "ring")):
                assert np.isfinite(want[k]).all(), k
                if k.endswith("velocity"):
                    assert np.abs(want[k]).max() > 1e-3, k
