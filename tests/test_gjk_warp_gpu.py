"""GJK on a warp (two shapes on its halves, hulls in registers, a repeated
state ending the loop) against the serial algorithm restated in Python
floats, which round like the device's -fmad=false double: the same pairs come
out separated, inside or going round, at vertex counts around the half-warp
and the 32 that registers hold, for poses from apart to just touching.  And
the horizon's edge cancellation against the serial add-or-erase list."""
import math

import numpy as np
import pytest

import rbps_b200
from rbps_b200 import abi, scenes

EPS = 1e-9


def dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def cross(a, b):
    return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])


def sub(a, b):
    return (a[0] - b[0], a[1] - b[1], a[2] - b[2])


def neg(a):
    return (-a[0], -a[1], -a[2])


def triple(a, b, c):
    return cross(cross(a, b), c)


def support(shape, d):
    kind, arg, pos = shape  # no rotation: quaternion arithmetic with an identity leaves every bit
    if kind == "hull":
        best = arg[0]
        bd = dot(best, d)
        for p in arg[1:]:
            x = dot(p, d)
            if x > bd:
                bd, best = x, p
        l = best
    else:
        n2 = dot(d, d)
        if n2 < EPS:
            l = (0.0, 0.0, 0.0)
        else:
            inv = 1.0 / math.sqrt(n2)
            l = (d[0] * inv * arg, d[1] * inv * arg, d[2] * inv * arg)
    return (pos[0] + l[0], pos[1] + l[1], pos[2] + l[2])


def gjk(A, B):
    """"valid" (apart), "inside" or "failed" (128 iterations)."""
    guess = sub(B[2], A[2])
    d = guess if dot(guess, guess) >= EPS else (1.0, 0.0, 0.0)

    def sup(x):
        return sub(support(A, x), support(B, neg(x)))

    s = [sup(d)]
    d = neg(s[0])
    for _ in range(128):
        w = sup(d)
        if dot(w, d) < 0.0:
            return "valid"
        s = [w] + s
        a, ao, ab = s[0], neg(s[0]), sub(s[1], s[0])
        if len(s) == 2:
            if dot(ab, ao) >= 0.0:
                d = triple(ab, ao, ab)
                if dot(d, d) < 1e-6:
                    x, y, z = (abs(v) for v in ab)
                    ax = (1.0, 0.0, 0.0) if x <= y and x <= z else ((0.0, 1.0, 0.0) if y <= z else (0.0, 0.0, 1.0))
                    d = cross(ab, ax)
                    if dot(d, d) < 1e-6:
                        d = cross(ab, (0.0, 0.0, 1.0))
            else:
                s, d = [a], ao
            continue
        ac = sub(s[2], a)
        abc = cross(ab, ac)

        def edge(v, e):
            return [a, v], triple(e, ao, e)

        def face(b, c, vb, vc, n, order):
            """Regions of triangle (a, b, c) with normal n."""
            if dot(cross(n, vc), ao) >= 0.0:
                if dot(vc, ao) >= 0.0:
                    return edge(c, vc)
                return edge(b, vb) if dot(vb, ao) >= 0.0 else ([a], ao)
            if dot(cross(vb, n), ao) >= 0.0:
                return edge(b, vb) if dot(vb, ao) >= 0.0 else ([a], ao)
            return order(n)

        if len(s) == 3:
            b, c = s[1], s[2]
            s, d = face(b, c, ab, ac, abc, lambda n: ([a, b, c], n) if dot(n, ao) >= 0.0 else ([a, c, b], neg(n)))
            continue
        b, c, e = s[1], s[2], s[3]
        ad = sub(e, a)
        acd, adb = cross(ac, ad), cross(ad, ab)
        info = (dot(abc, ao) > 1e-10) + 2 * (dot(acd, ao) > 1e-10) + 4 * (dot(adb, ao) > 1e-10)
        if info == 0:
            return "inside"
        if info == 1:
            s, d = face(b, c, ab, ac, abc, lambda n: ([a, b, c], n))
        elif info == 2:
            s, d = face(c, e, ac, ad, acd, lambda n: ([a, c, e], n))
        elif info == 4:
            s, d = face(e, b, ad, ab, adb, lambda n: ([a, e, b], n))
        elif info in (3, 5, 6):
            v, x = {3: (c, ac), 5: (b, ab), 6: (e, ad)}[info]
            s, d = edge(v, x) if dot(x, ao) >= 0.0 else ([a], ao)
        else:
            s, d = [a], ao
    return "failed"


def _hull(rng, n):
    d = rng.standard_normal((n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.3, 0.8, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("nv", [4, 15, 16, 17, 31, 32, 33, 70])
def test_gjk_decides_as_serial(rbps, nv):
    rng = np.random.default_rng(nv)
    b = rbps.Batch(1, 1.0 / 60.0, 1, abi.PRECISION_FP64)
    pts = [_hull(rng, nv), _hull(rng, 20)]
    ids = [b.add_hull(p, rbps_b200.quickhull(p)) for p in pts]
    b.add_world(0, scenes.small_world(0, 1))
    b.commit()
    n = 400
    ca, cb = np.zeros(n, abi.COLLIDER_DT), np.zeros(n, abi.COLLIDER_DT)
    ta, tb = np.zeros((n, 7)), np.zeros((n, 7))
    ta[:, 3] = tb[:, 3] = 1.0
    pairs = []
    for k in range(n):
        ball = k % 2 == 0
        r = float(rng.uniform(0.2, 0.5))
        u = rng.standard_normal(3)
        u /= np.linalg.norm(u)
        # how far apart the shapes reach along u, then a little more or less
        reach = (pts[0] @ u).max() + (r if ball else (pts[1] @ -u).max())
        pos = u * (reach + rng.choice([-0.3, -1e-2, -1e-6, 0.0, 1e-6, 1e-2]))
        ca[k]["shape"] = cb[k]["shape"] = abi.SHAPE_CONVEX_HULL
        ca[k]["hull"] = ids[0]
        cb[k]["hull"] = ids[1]
        other = ("hull", [tuple(p) for p in pts[1]], tuple(pos))
        if ball:
            cb[k]["shape"] = abi.SHAPE_SPHERE
            cb[k]["params"][0] = r
            other = ("sphere", r, tuple(pos))
        tb[k, :3] = pos
        pairs.append((("hull", [tuple(p) for p in pts[0]], (0.0, 0.0, 0.0)), other))
    want = [gjk(*p) for p in pairs]
    got = b.collide(ca, ta, cb, tb)["status"] == abi.COLLIDE_HIT
    for k, w in enumerate(want):
        assert w == "inside" or not got[k], (k, w)
    inside = np.array([w == "inside" for w in want])
    assert inside.sum() > 50 and got[inside].mean() > 0.9  # EPA gives up on a few of the grazing ones


def test_horizon_model():
    """warp_horizon: an edge met an odd number of times stands where it was
    met last."""
    rng = np.random.default_rng(3)
    for n, m in ((0, 2), (3, 3), (31, 4), (96, 5), (300, 9)):
        edges = [tuple(rng.choice(m, 2, replace=False)) for _ in range(n)]
        serial = []
        for e in edges:
            hit = next((i for i, f in enumerate(serial) if f in (e, e[::-1])), None)
            if hit is None:
                serial.append(e)
            else:
                del serial[hit]
        key = [tuple(sorted(e)) for e in edges]
        warp = [e for i, e in enumerate(edges) if key.count(key[i]) % 2 and i == max(j for j, k in enumerate(key) if k == key[i])]
        assert warp == serial
