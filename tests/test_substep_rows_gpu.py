"""Both float substep kernels (three resident CTAs an SM, and four) give the
same bits for every kind of row: contacts of all shapes, and damped, limited
and driven joints of each type.  The same worlds step alone and among enough
others that the launch no longer fits three CTAs an SM."""
import numpy as np
import pytest

from rbps_b200 import abi, scenes
from test_joint_states_gpu import jointed_worlds

pytestmark = pytest.mark.gpu

MAKERS = {
    "joints": lambda: [spec for _, spec in jointed_worlds()],
    "hulls": lambda: [scenes.hull_world(seed=1, n=24), scenes.round_world(seed=2, n=24)],
    "triangles": lambda: [scenes.terrain_world(seed=3, n=24), scenes.mesh_world(seed=4, n=24)],
    "capsules": lambda: [scenes.capsule_world(seed=5, n=48), scenes.chain_world(seed=6, n_bodies=60, damping=1.0)],
}


@pytest.mark.parametrize("precision", [abi.PRECISION_FP32, abi.PRECISION_FP32_POS64])
@pytest.mark.parametrize("name", sorted(MAKERS))
def test_few_and_many_agree(rbps, name, precision):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    few = MAKERS[name]()
    filler = [scenes.small_world(seed=0, n=4)] * (3 * sms + 8)
    states = []
    for worlds in (few, few + filler):
        b = rbps.Batch.from_scene(scenes.Scene(name, 1.0 / 60.0, 4, 0, worlds), precision, abi.SOLVE_COLORED)
        b.set_launch(team_bodies=1, pair_bodies=1)  # a CTA a world
        b.set_state_check(False)
        b.step(20)
        states.append([b.state(w) for w in range(len(few))])
    for w, (a, c) in enumerate(zip(*states)):
        for f in a:
            np.testing.assert_array_equal(a[f], c[f], err_msg="%d %s" % (w, f))
