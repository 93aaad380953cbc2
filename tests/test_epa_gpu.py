"""EPA on a warp (faces and horizon split over its lanes, edges cancelled in
parallel) against the serial algorithm (EPA.cpp:141-378) restated in Python
floats, which round like the device's -fmad=false double: hit or not, depth,
normal and contact point are the same bits.  The shapes carry no polygon
tables or meet a sphere, so a manifold is EPA's own point.  Among the pairs
are ones whose GJK goes round for good (the device stops them at the first
repeated state), ones that run out of faces, and horizons of more than 32
edges, a warp's width."""
import math

import numpy as np
import pytest

from rbps_b200 import abi, scenes
from test_gjk_warp_gpu import EPS, cross, dot, neg, sub, support, triple

MAX_FACES, MAX_VERTS, MAX_ITER = 256, 128, 128


def scale(a, s):
    return (a[0] * s, a[1] * s, a[2] * s)


def add(a, b):
    return (a[0] + b[0], a[1] + b[1], a[2] + b[2])


def point(A, B, d):
    """A's support, B's and their difference along d."""
    a, b = support(A, d), support(B, neg(d))
    return a, b, sub(a, b)


def gjk(A, B):
    """("apart" | "inside" | "round", simplex): the serial loop (GJK.cpp:18-97),
    128 iterations at most, the simplex's points newest first."""
    guess = sub(B[2], A[2])
    d = guess if dot(guess, guess) >= EPS else (1.0, 0.0, 0.0)
    s = [point(A, B, d)]
    d = neg(s[0][2])
    for _ in range(128):
        w = point(A, B, d)
        if dot(w[2], d) < 0.0:
            return "apart", s
        s = [w] + s
        a = w[2]
        ao = neg(a)
        to = [sub(p[2], a) for p in s]  # to[1]: from the newest to the one before it

        def edge(i):
            """Keeps the newest and point i, or the newest alone."""
            if dot(to[i], ao) >= 0.0:
                return [s[0], s[i]], triple(to[i], ao, to[i])
            return [s[0]], ao

        def face(i, j, both):
            """The regions of triangle (newest, i, j)."""
            n = cross(to[i], to[j])
            if dot(cross(n, to[j]), ao) >= 0.0:
                return edge(j) if dot(to[j], ao) >= 0.0 else edge(i)
            if dot(cross(to[i], n), ao) >= 0.0:
                return edge(i)
            if both and dot(n, ao) < 0.0:
                return [s[0], s[j], s[i]], neg(n)
            return [s[0], s[i], s[j]], n

        if len(s) == 2:
            s, d = edge(1)
            if len(s) == 2 and dot(d, d) < 1e-6:  # the origin on the line: any direction off it
                x, y, z = (abs(v) for v in to[1])
                ax = (1.0, 0.0, 0.0) if x <= y and x <= z else ((0.0, 1.0, 0.0) if y <= z else (0.0, 0.0, 1.0))
                d = cross(to[1], ax)
                if dot(d, d) < 1e-6:
                    d = cross(to[1], (0.0, 0.0, 1.0))
        elif len(s) == 3:
            s, d = face(1, 2, True)
        else:
            out = [dot(cross(to[i], to[j]), ao) > 1e-10 for i, j in ((1, 2), (2, 3), (3, 1))]
            if not any(out):
                return "inside", s
            if sum(out) == 3:
                s, d = [s[0]], ao
            elif sum(out) == 2:
                s, d = edge({(0, 1): 2, (0, 2): 1, (1, 2): 3}[tuple(k for k in range(3) if out[k])])
            else:
                i, j = ((1, 2), (2, 3), (3, 1))[out.index(True)]
                s, d = face(i, j, False)
    return "round", s


def face_normal(V, v):
    """(normal, distance, centroid) of face v, or None (EPA.cpp:19-67)."""
    a, b, c = (V[i][2] for i in v)
    n = cross(sub(b, a), sub(c, a))
    ln = math.sqrt(dot(n, n))
    if ln < EPS:
        return None
    n = scale(n, 1.0 / ln)
    d = dot(n, a)
    if d < -1e-12:
        n, d = neg(n), -d
    elif d <= 1e-12:
        t = next((t for t in (dot(n, p[2]) for p in V) if abs(t) > 1e-12), None)
        if t is None:
            return None
        if t > 1e-12:
            n = neg(n)
        d = 0.0
    return n, d, scale(add(add(a, b), c), 1.0 / 3.0)


def epa(A, B, seed, note):
    """(normal, depth, contact) or None.  seed: the tetrahedron's points
    (on A, on B, difference), newest first."""
    V = list(seed)
    a, b, c, e = (p[2] for p in V)
    pn = cross(sub(b, a), sub(c, a))
    if dot(pn, pn) < EPS * EPS:
        pn = cross(sub(b, a), sub(e, a))
    if dot(pn, pn) < EPS * EPS:
        pn = cross(sub(c, a), sub(e, a))
    if dot(pn, pn) > EPS * EPS:
        n2 = dot(pn, pn)
        pn = scale(pn, 1.0 / math.sqrt(n2)) if n2 >= EPS else (0.0, 0.0, 0.0)
        if abs(dot(sub(e, a), pn)) < 1e-5:
            pos, opp = (dot(sub(point(A, B, x)[2], a), x) for x in (pn, neg(pn)))
            if pos < 1e-4 or opp < 1e-4:
                w = add(add(add(V[0][0], V[1][0]), V[2][0]), V[3][0])
                return pn if pos <= opp else neg(pn), 0.0, scale(w, 0.25)
    F = []
    for v in ((0, 1, 2), (0, 2, 3), (0, 3, 1), (1, 2, 3)):
        f = face_normal(V, v)
        if f is None:
            return None
        F.append([v, *f, True])
    for _ in range(MAX_ITER):
        live = [f for f in F if f[4]]
        if not live:
            return None
        face = min(live, key=lambda f: f[2])  # the first of the nearest
        v, n, d, _, _ = face
        w = point(A, B, n)
        grown = dot(w[2], n) - d >= 1e-6
        if not grown:
            q = scale(n, d)
            p0, p1, p2 = (V[i][2] for i in v)
            e0, e1, r = sub(p1, p0), sub(p2, p0), sub(q, p0)
            d00, d01, d11, d20, d21 = dot(e0, e0), dot(e0, e1), dot(e1, e1), dot(r, e0), dot(r, e1)
            den = d00 * d11 - d01 * d01
            at = V[v[0]][0]
            if abs(den) >= EPS:
                s = (d11 * d20 - d01 * d21) / den
                t = (d00 * d21 - d01 * d20) / den
                at = add(add(scale(V[v[0]][0], 1.0 - s - t), scale(V[v[1]][0], s)), scale(V[v[2]][0], t))
            return n, d, at
        if any(dot(x, x) < EPS * EPS for x in (sub(p[2], w[2]) for p in V)):
            return n, d, V[v[0]][0]
        if len(V) >= MAX_VERTS:
            return None
        V.append(w)
        edges, seen = [], 0
        for f in F:
            if f[4] and dot(f[1], sub(w[2], f[3])) > 0.0:
                f[4] = False
                seen += 1
                for x, y in zip(f[0], f[0][1:] + f[0][:1]):
                    hit = next((i for i, z in enumerate(edges) if z in ((x, y), (y, x))), None)
                    if hit is None:
                        edges.append((x, y))
                    else:
                        del edges[hit]
        note["edges"] = max(note.get("edges", 0), 3 * seen)
        note["kept"] = max(note.get("kept", 0), len(edges))
        for x, y in edges:
            if len(F) >= MAX_FACES:
                note["out"] = True
                return None
            v = (x, y, len(V) - 1)
            f = face_normal(V, v)
            if f is not None:
                F.append([v, *f, True])
    return None


def model(A, B, note):
    """What the device's test gives: None, or (normal, depth, contact)."""
    note["gjk"], simplex = gjk(A, B)
    return epa(A, B, simplex, note) if note["gjk"] == "inside" else None


def cloud(rng, n, axes):
    d = rng.standard_normal((n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True) * np.asarray(axes)


def needle(rng):
    return np.concatenate([cloud(rng, int(rng.integers(8, 200)), (0.05, 0.05, 0.05)), [[0.0, 1.0, 0.0], [0.01, -1.0, 0.0]]])


def ring(rng):
    """A many-sided prism with a spike, turned at random: a new vertex sees
    many of its faces."""
    n = int(rng.integers(8, 200))
    t, h = np.arange(n) * 2.0 * np.pi / n, np.exp(rng.uniform(-5.0, -1.0))
    p = np.concatenate([np.stack([np.cos(t), 0.0 * t + y, np.sin(t)], 1) for y in (h, -h)] +
                       [[[0.0, rng.uniform(0.2, 2.0), 0.0]]])
    return p @ np.linalg.qr(rng.standard_normal((3, 3)))[0]


def pairs(family, rng, n):
    """n pairs of (points of A, points of B or a radius, position of B)."""
    for _ in range(n):
        if family == "needles":
            yield needle(rng), ring(rng), rng.standard_normal(3) * np.exp(rng.uniform(-6.0, 0.0))
            continue
        a = cloud(rng, int(rng.choice([4, 15, 16, 17, 31, 32, 33, 70, 200])), np.exp(rng.uniform(-1.5, 0.0, 3)))
        u = rng.standard_normal(3)
        u /= np.linalg.norm(u)
        if family == "balls":  # around touching, where GJK goes round, and deeper, where EPA may not end
            r = float(rng.uniform(0.2, 0.5))
            off = rng.choice([-0.3, -0.1, -1e-3, -1e-6, -1e-8, 0.0, 1e-8, 1e-6])
            yield a, r, a[np.argmax(a @ u)] + u * (r + off)
        else:
            yield a, cloud(rng, int(rng.integers(4, 80)), np.exp(rng.uniform(-1.5, 0.0, 3))), u * rng.uniform(0.0, 0.8)


def models(family, n):
    rng = np.random.default_rng(7)
    out = []
    for a, b, pos in pairs(family, rng, n):
        sa = ("hull", [tuple(map(float, p)) for p in a], (0.0, 0.0, 0.0))
        at = tuple(map(float, pos))
        sb = ("sphere", b, at) if family == "balls" else ("hull", [tuple(map(float, p)) for p in b], at)
        note = {}
        out.append((a, b, at, model(sa, sb, note), note))
    return out


FAMILIES = {"balls": 300, "clouds": 200, "needles": 300}


def test_model_meets_the_hard_cases():
    """The pairs below include every way out, and horizons past a warp."""
    notes = {f: [m[4] for m in models(f, n)] for f, n in FAMILIES.items()}
    assert sum(x["gjk"] == "round" for x in notes["balls"]) >= 5
    assert sum(x.get("out", False) for x in notes["balls"]) >= 1
    assert sum(x.get("edges", 0) > 32 for x in notes["needles"]) >= 5
    for f in FAMILIES:
        assert sum(x["gjk"] == "inside" for x in notes[f]) >= 50
        assert sum(x["gjk"] == "apart" for x in notes[f]) >= 5


@pytest.mark.gpu
@pytest.mark.parametrize("family", sorted(FAMILIES))
def test_epa_as_serial(rbps, family):
    cases = models(family, FAMILIES[family])
    n = len(cases)
    b = rbps.Batch(1, 1.0 / 60.0, 1, abi.PRECISION_FP64)
    ca, cb = np.zeros(n, abi.COLLIDER_DT), np.zeros(n, abi.COLLIDER_DT)
    ta, tb = np.zeros((n, 7)), np.zeros((n, 7))
    ta[:, 3] = tb[:, 3] = 1.0
    none = np.zeros((0, 3), np.uint32)  # no triangles, no polygon tables
    ca["shape"] = cb["shape"] = abi.SHAPE_CONVEX_HULL
    for k, (pa, pb, at, _, _) in enumerate(cases):
        ca[k]["hull"] = b.add_hull(pa, none)
        if family == "balls":
            cb[k]["shape"] = abi.SHAPE_SPHERE
            cb[k]["params"][0] = pb
        else:
            cb[k]["hull"] = b.add_hull(pb, none)
        tb[k, :3] = at
    b.add_world(0, scenes.small_world(0, 1))
    b.commit()
    got = b.collide(ca, ta, cb, tb)
    for k, (_, _, _, want, note) in enumerate(cases):
        assert (got["status"][k] == abi.COLLIDE_HIT) == (want is not None), (k, note)
        if want is None:
            continue
        normal, depth, contact = want
        assert got["n_points"][k] == 1
        np.testing.assert_array_equal(got["depth"][k, 0], depth, err_msg=str((k, note)))
        np.testing.assert_array_equal(got["normal"][k], normal, err_msg=str((k, note)))
        np.testing.assert_array_equal(got["position"][k, 0], contact, err_msg=str((k, note)))
