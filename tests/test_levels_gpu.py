"""The reference's contact order relaxed level by level (schedule_levels):
the same bits whichever team steps the world (a CTA, half a CTA, a warp;
bodies in shared memory or in place; level offsets in shared memory or in
the world's scratch), and the compiled reference's bits where it is present.
"""
import numpy as np
import pytest

from helpers import bit_equal
from rbps_b200 import abi, scenes

pytestmark = pytest.mark.gpu

WORLDS = {
    "empty_contacts": lambda: scenes.small_world(seed=1, n=1),
    "one_chunk": lambda: scenes.small_world(seed=2, n=32, hi=(2.0, 3.0, 2.0), lo=(-2.0, 0.3, -2.0)),
    "many_chunks": lambda: scenes.small_world(seed=3, n=400, hi=(4.0, 6.0, 4.0), lo=(-4.0, 0.3, -4.0)),
    "chains": lambda: scenes.chain_world(seed=4, n_bodies=90),
    # a stack: a level for almost every contact, more than the shared words hold
    "stack": lambda: scenes.config4(seed=5, n_worlds=1, height=200, offset=0.0, mass_ratio=1.0).worlds[0],
    # beyond the shared-memory world copies
    "large": lambda: scenes.small_world(seed=6, n=1100),
}
TEAMS = [{}, {"team_bodies": 1, "pair_bodies": 1}, {"team_bodies": 5000, "pair_bodies": 2},
         {"team_bodies": 5000, "pair_bodies": 5000}]


@pytest.mark.parametrize("name", sorted(WORLDS))
def test_teams_agree(rbps, name):
    spec = WORLDS[name]()
    states = []
    for team in TEAMS:
        b = rbps.Batch.from_scene(scenes.Scene(name, 1.0 / 60.0, 3, 4, [spec]), abi.PRECISION_FP64,
                                  abi.SOLVE_REFERENCE_ORDER, max_pairs_per_world=1 << 16)
        if team:
            b.set_launch(**team)
        b.step(4)
        states.append(b.state(0))
    for st in states[1:]:
        for f in st:
            np.testing.assert_array_equal(st[f], states[0][f], err_msg=f)


@pytest.mark.parametrize("name", sorted(WORLDS))
def test_live_oracle(rbps, ref, name):
    spec = WORLDS[name]()
    w_ref = ref.RefWorld(spec, 1.0 / 60.0, 3)
    b = rbps.Batch.from_scene(scenes.Scene(name, 1.0 / 60.0, 3, 4, [spec]), abi.PRECISION_FP64,
                              abi.SOLVE_REFERENCE_ORDER, max_pairs_per_world=1 << 16)
    for _ in range(4):
        w_ref.step(1)
        b.step(1)
        assert bit_equal(b.state(0), w_ref.state())
