"""The float substep kernel compiled for three resident CTAs (launches that
fit them) and for four (larger ones) gives a world the same bits, and so do
narrowphase ranges of one chunk and of many."""
import numpy as np
import pytest

from rbps_b200 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PRECISION_FP32, abi.PRECISION_FP64])
@pytest.mark.parametrize("count", [1, 8])
def test_few_and_many_worlds_agree(rbps, precision, count):
    n = 460  # a CTA a world: more CTAs than three an SM on 148 SMs
    sc = scenes.config3(seed=5, n_worlds=n, lo_bodies=8, hi_bodies=16)
    few = scenes.Scene(sc.name, sc.timestep, sc.substeps, 0, sc.worlds[:count])
    states = []
    for scene in (sc, few):
        b = rbps.Batch.from_scene(scene, precision, abi.SOLVE_COLORED)
        b.set_launch(team_bodies=1, pair_bodies=1)
        b.set_state_check(False)
        b.step(40)
        states.append([b.state(w) for w in range(count)])
    for a, c in zip(*states):
        for f in a:
            np.testing.assert_array_equal(a[f], c[f], err_msg=f)
