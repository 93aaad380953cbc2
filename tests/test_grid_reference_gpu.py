"""The reference's order on the cooperative grid (more than 4,096 bodies):
clusters that never meet, in one large world, take the states of the same
clusters as worlds of their own, which step on a CTA each.  In double every
bit agrees: a cluster's contacts keep their order among themselves, and
levels, rows and joints are the same operations on either team."""
import numpy as np
import pytest

from rbps_b200 import abi, scenes

pytestmark = pytest.mark.gpu


def cluster(k, n=460, damping=0.0):
    """Bodies above the ground at x about 60 k, with two revolute chains."""
    x = 60.0 * k
    rng = np.random.default_rng(k)
    bodies, forces, colliders = scenes.box_sphere_world(rng, n, lo=(x - 4.0, 0.3, -4.0), hi=(x + 4.0, 7.0, 4.0))
    joints = []
    for z in (-9.0, 9.0):
        scenes.capsule_chain(bodies, forces, colliders, joints, (x - 4.0, 1.0 + k % 3, z), damping=damping)
    return bodies, forces, colliders, joints


def union(parts):
    """One world of all the parts, whose body 0 is the same ground."""
    bodies, forces, colliders, joints = [], [], [], []
    for k, (b, f, c, j) in enumerate(parts):
        skip = 0 if k == 0 else 1
        base = len(bodies) - skip
        bodies += b[skip:]
        forces += f[skip:]
        for col in c[skip:]:
            col = col.copy()
            col["body_id"] += base
            colliders.append(col)
        for jt in j:
            jt = jt.copy()
            jt["body_1"] += base
            jt["body_2"] += base
            joints.append(jt)
    return scenes._finish(bodies, forces, colliders, joints)


@pytest.mark.parametrize("damping", [0.0, 2.0])
def test_grid_equals_ctas(rbps, damping):
    parts = [cluster(k, damping=damping) for k in range(9)]
    one = scenes.Scene("one", 1.0 / 60.0, 4, 0, [union(parts)])
    assert one.n_bodies > 4096
    many = scenes.Scene("many", 1.0 / 60.0, 4, 0, [scenes._finish(*p) for p in parts])
    states = []
    for sc in (one, many):
        b = rbps.Batch.from_scene(sc, abi.PRECISION_FP64, abi.SOLVE_REFERENCE_ORDER, max_pairs_per_world=1 << 17)
        b.set_state_check(False)
        b.step(6)
        states.append([b.state(w) for w in range(len(sc.worlds))])
    big = states[0][0]
    at = 1
    for st in states[1]:
        n = len(st["position"]) - 1
        for f in st:
            np.testing.assert_array_equal(big[f][at:at + n], st[f][1:], err_msg=f)
        assert np.isfinite(st["position"]).all()
        at += n
    assert at == one.n_bodies
