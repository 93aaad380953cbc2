"""The general sweep (sweep_runs) against the restated broadphase
(oracle/sap.py), pair order included: runs shorter and longer than a warp's
32, more hits than a warp stages, groups on both sides of the size from which
they are radix sorted, ties, and boxes with infinite or NaN sides."""
import numpy as np
import pytest

from oracle.sap import SapBroadPhase

pytestmark = pytest.mark.gpu

TEAMS = [(False, 256), (True, 256), (True, 32)]


def _boxes(name):
    rng = np.random.default_rng(len(name))
    if name == "spread":  # a few partners each
        lo = rng.uniform(0, 60, (700, 3)) * (1, 0.1, 0.1)
        return np.concatenate([lo, lo + rng.uniform(0.2, 1.0, (700, 3))], 1)
    if name.startswith("pile"):  # every box meets every other: groups of 0 .. n - 1
        n = int(name[4:])
        lo = rng.uniform(0, 1, (n, 3))
        return np.concatenate([lo, lo + 2.0], 1)
    if name == "ties":  # a lattice: equal endpoints on every axis
        g = np.stack(np.meshgrid(*[np.arange(7.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
        return np.concatenate([g, g + 0.9], 1)
    lo = rng.uniform(0, 8, (90, 3))
    b = np.concatenate([lo, lo + 1.0], 1)
    b[3, 3:] = np.inf
    b[11, :3] = -np.inf
    b[20, 1] = b[20, 4] = np.nan
    b[31, 4] = 1e300
    b[40, 1] = -1e300
    return b


@pytest.mark.parametrize("team", TEAMS, ids=lambda t: f"{'cta' if t[0] else 'grid'}{t[1]}")
@pytest.mark.parametrize("name", ["spread", "pile2", "pile33", "pile65", "pile66", "pile300", "ties", "wild"])
def test_pairs_in_order(rbps, name, team):
    boxes = _boxes(name)
    g, r = rbps.BroadPhase(single_cta=team[0], block=team[1]), SapBroadPhase()
    for k, b in enumerate(boxes):
        g.insert(k, b)
        r.insert(k, b)
    for turn in range(2):
        g.update()
        r.update()
        want = np.array(r.pairs, np.uint32).reshape(-1, 2)
        assert len(want) > 0
        np.testing.assert_array_equal(g.pairs(), want)
        for k in range(0, len(boxes), 5):  # some move, then again
            g.move(k, boxes[k] + 0.7)
            r.move(k, boxes[k] + 0.7)
