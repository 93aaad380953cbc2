"""Coloured runs repeat bit for bit where a body has more contacts than there
are colours: a plate that more than 128 balls rest on, so that contacts go to
the serial colour in every substep, some past the second-level colours too.
In small worlds (bodies in shared memory, and in place) and in a large one,
where most bodies touch nothing."""
import numpy as np
import pytest

from rbps_b200 import abi, scenes

pytestmark = pytest.mark.gpu

FIELDS = ("position", "orientation", "linear_velocity", "angular_velocity")


def scene(n, gap, side=16):
    """Ground, a plate with side^2 balls `gap` above it, a column of balls
    that touch, and n balls in free fall."""
    rng = np.random.default_rng(1)
    bodies, forces, colliders = [], [], []
    scenes._ground(bodies, colliders, forces, 0.5, 0.0)

    def put(pos, shape, params, mass):
        b, f = scenes._dyn_body(pos, (1.0, 0.0, 0.0, 0.0), *mass)
        colliders.append(scenes._collider(shape, params, len(bodies), 0.5, 0.0))
        bodies.append(b)
        forces.append(f)

    h = (0.6 * side, 0.2, 0.6 * side)
    put((0.0, 0.19, 0.0), abi.SHAPE_BOX, h, scenes.box_mass(h))
    for k in range(side * side):
        x, z = 1.1 * (k % side - (side - 1) / 2), 1.1 * (k // side - (side - 1) / 2)
        r = float(rng.uniform(0.3, 0.4))
        put((x, 0.39 + r + gap, z), abi.SHAPE_SPHERE, (r,), scenes.sphere_mass(r))
    # their order shows in the state, and their bodies' words lie among the balls'
    for k in range(12):
        put((-20.0, 0.39 + 0.78 * k, 0.03 * (k % 3)), abi.SHAPE_SPHERE, (0.4,), scenes.sphere_mass(0.4))
    for k in range(n):
        put((3.0 * (k % 65) + 30.0, 50.0, 3.0 * (k // 65)), abi.SHAPE_SPHERE, (0.3,), scenes.sphere_mass(0.3))
    return scenes.Scene("plate", 1.0 / 60.0, 1, 0, [scenes._finish(bodies, forces, colliders, [])])


SIZES = [0, 1500, 4200]  # in shared memory, in place, on the grid


@pytest.mark.parametrize("precision", [abi.PRECISION_FP32, abi.PRECISION_FP64])
@pytest.mark.parametrize("n", SIZES)
def test_runs_agree(rbps, n, precision):
    """The first substep of fresh batches, whose history is the same: the
    order within the serial colour is the list's."""
    states = []
    for _ in range(6):
        b = rbps.Batch.from_scene(scene(n, -0.01), precision, abi.SOLVE_COLORED)
        b.step(1)
        assert b.stats()["serial_overflow"] > 128
        states.append(b.state_all(FIELDS))
    for st in states[1:]:
        for f in FIELDS:
            np.testing.assert_array_equal(st[f], states[0][f], err_msg=f)


@pytest.mark.parametrize("precision", [abi.PRECISION_FP32, abi.PRECISION_FP64])
@pytest.mark.parametrize("n", SIZES)
def test_restored_run_repeats(rbps, n, precision):
    """Whatever was coloured before: the colouring starts from cleared
    counters, of the contacting bodies alone where they are few.  Here the
    column's contacts are coloured before the balls land, and again after a
    run in which they have."""
    b = rbps.Batch.from_scene(scene(n, 0.02), precision, abi.SOLVE_COLORED)
    slot = b.snapshot()
    runs = []
    for _ in range(3):
        b.restore(slot)
        b.step(1)
        assert b.stats()["serial_overflow"] == 0 and b.stats()["contacts"] > 8
        b.step(9)
        assert b.stats()["serial_overflow"] > 0
        runs.append(b.state_all(FIELDS))
    for st in runs[1:]:
        for f in FIELDS:
            np.testing.assert_array_equal(st[f], runs[0][f], err_msg=f)


@pytest.mark.parametrize("precision", [abi.PRECISION_FP32, abi.PRECISION_FP64])
def test_launch_shapes_agree(rbps, precision):
    """A CTA, half a CTA and a warp relax the serial colour in one order."""
    states = []
    for team, pair in ((1, 1), (5000, 2), (5000, 5000)):
        b = rbps.Batch.from_scene(scene(0, -0.01), precision, abi.SOLVE_COLORED)
        b.set_launch(team_bodies=team, pair_bodies=pair)
        b.step(1)
        assert b.stats()["serial_overflow"] > 128
        b.step(3)
        states.append(b.state_all(FIELDS))
    for st in states[1:]:
        for f in FIELDS:
            np.testing.assert_array_equal(st[f], states[0][f], err_msg=f)
