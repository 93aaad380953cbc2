"""rbps_batch_set_state followed at once by a read, or by a step: both run on
the batch's stream behind the upload, whichever fields it wrote."""
import numpy as np
import pytest

from rbps_b200 import abi, scenes

pytestmark = pytest.mark.gpu

FIELDS = ("position", "orientation", "linear_velocity", "angular_velocity")


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_FP32])
@pytest.mark.parametrize("n", [30, 20000])
def test_set_then_get(rbps, precision, n):
    spec = scenes.small_world(seed=2, n=n, lo=(-60.0, 1.0, -60.0), hi=(60.0, 90.0, 60.0))
    b = rbps.Batch.from_scene(scenes.Scene("set", 1.0 / 60.0, 1, 0, [spec]), precision, abi.SOLVE_COLORED)
    kind = np.float64 if precision == abi.PRECISION_FP64 else np.float32
    rng = np.random.default_rng(n)
    held = b.state(0)
    for k in range(20):
        fields = [f for i, f in enumerate(FIELDS) if k % 4 == i or k % 3 == 0]
        for f in fields:
            held[f] = rng.standard_normal(held[f].shape).astype(kind).astype(np.float64)
        b.set_state(0, {f: held[f] for f in fields})
        got = b.state(0)
        for f in FIELDS:
            np.testing.assert_array_equal(got[f], held[f], err_msg="%d %s" % (k, f))


def test_set_then_step(rbps):
    """A state set just before a step is the one that is stepped."""
    spec = scenes.small_world(seed=2, n=20000, lo=(-60.0, 1.0, -60.0), hi=(60.0, 90.0, 60.0))
    sc = scenes.Scene("set", 1.0 / 60.0, 1, 0, [spec])
    states = []
    for _ in range(2):
        b = rbps.Batch.from_scene(sc, abi.PRECISION_FP64, abi.SOLVE_COLORED)
        rng = np.random.default_rng(1)
        for _ in range(5):
            v = rng.standard_normal((20001, 3))
            v[0] = 0.0
            b.set_state(0, {"linear_velocity": v})
            b.step(1)
            if not states:
                b.synchronize()
        states.append(b.state(0))
    for f in FIELDS:
        np.testing.assert_array_equal(states[1][f], states[0][f], err_msg=f)
