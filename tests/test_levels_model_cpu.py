"""The level schedule of the reference order, on the CPU: levels_warp's
32-at-a-time arithmetic restated in numpy gives the serial definition, and
relaxing level by level gives the serial walk's result."""
import numpy as np
import pytest


def serial_levels(a, b, dyn, n_bodies):
    last = np.zeros(n_bodies, int)
    out = []
    for x, y in zip(a, b):
        l = max(last[x] if dyn[x] else 0, last[y] if dyn[y] else 0)
        for k in (x, y):
            if dyn[k]:
                last[k] = l + 1
        out.append(l)
    return np.array(out, int)


def warp_levels(a, b, dyn, n_bodies):
    last = np.zeros(n_bodies, int)
    out = np.zeros(len(a), int)
    for k0 in range(0, len(a), 32):
        m = min(32, len(a) - k0)
        A, B = a[k0:k0 + m], b[k0:k0 + m]
        l = np.maximum(np.where(dyn[A], last[A], 0), np.where(dyn[B], last[B], 0))
        last_a, last_b = dyn[A].copy(), dyn[B].copy()
        lane = np.arange(m)
        for j in range(m):
            on_a = dyn[A] & ((A[j] == A) | (B[j] == A))
            on_b = dyn[B] & ((A[j] == B) | (B[j] == B))
            l = np.where((j < lane) & (on_a | on_b), np.maximum(l, l[j] + 1), l)
            last_a &= ~((j > lane) & on_a)
            last_b &= ~((j > lane) & on_b)
        assert len(set(A[last_a]) & set(B[last_b])) == 0 and len(set(A[last_a])) == last_a.sum()
        last[A[last_a]] = l[last_a] + 1
        last[B[last_b]] = l[last_b] + 1
        out[k0:k0 + m] = l
    return out


@pytest.mark.parametrize("n,n_bodies", [(0, 2), (1, 2), (31, 5), (32, 40), (33, 3), (64, 200), (501, 60)])
def test_levels(n, n_bodies):
    rng = np.random.default_rng(n)
    a = rng.integers(0, n_bodies, n)
    b = (a + rng.integers(1, n_bodies, n)) % n_bodies
    dyn = rng.random(n_bodies) < 0.8
    lv = warp_levels(a, b, dyn, n_bodies)
    np.testing.assert_array_equal(lv, serial_levels(a, b, dyn, n_bodies))
    # an update that does not commute: the order on every body must be kept

    def relax(order):
        x = np.arange(1, n_bodies + 1, dtype=object)
        for q in order:
            h = hash((q, x[a[q]], x[b[q]]))
            for k in (a[q], b[q]):
                if dyn[k]:
                    x[k] = hash((h, k))
        return list(x)

    shuffled = sorted(range(n), key=lambda q: (lv[q], -q))
    assert relax(range(n)) == relax(shuffled)
