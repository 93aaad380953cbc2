"""A pair table that is too small keeps the same pairs in every run: those of
the earliest opening endpoints, in the sweep's order (the sweep in global
memory: more objects than a CTA stages, and a large world's grid)."""
import numpy as np
import pytest

from rbps_b200 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [900, 4500])
@pytest.mark.parametrize("share", [0.0, 0.3, 0.999])
def test_kept_pairs(rbps, n, share):
    edge = 1.5 * n ** (1.0 / 3.0) / 2.0
    spec = scenes.small_world(seed=n, n=n, lo=(-edge, 1.0, -edge), hi=(edge, 1.0 + 2.0 * edge, edge))
    sc = scenes.Scene("dense", 1.0 / 60.0, 1, 0, [spec])

    def pairs(cap):
        b = rbps.Batch.from_scene(sc, abi.PRECISION_FP64, abi.SOLVE_COLORED, max_pairs_per_world=cap)
        b.set_dump(True)
        b.step(1)
        if cap < 1 << 16:
            with pytest.raises(rbps.RbpsError) as e:
                b.synchronize()
            assert e.value.code == abi.ERR_CAPACITY
        return b.pairs(0), b.sap_state(0)[1], b.state(0)

    full, ids, _ = pairs(1 << 16)
    opens = np.zeros(n, np.int64)  # position of each object's opening endpoint
    opens[ids[ids % 2 == 0] // 2] = np.flatnonzero(ids % 2 == 0)
    at = np.sort(opens[full.astype(np.int64) - 1], axis=1)  # collider 0 is the ground plane, not a SAP object
    np.testing.assert_array_equal(np.lexsort((at[:, 0], at[:, 1])), np.arange(len(full)))
    cap = max(1, int(share * len(full)))
    first = np.lexsort((at[:, 1], at[:, 0]))[:cap]  # by the earlier object, then the later
    want = full[np.sort(first)]
    kept = [pairs(cap) for _ in range(3)]
    for got, _, st in kept:
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(st["position"], kept[0][2]["position"])
