"""Writes states.npz beside this file from the rbps_b200 that is imported.

    PYTHONPATH=<tree> python tests/golden/joints/record.py

The committed file is of commit 3d69e2e, whose kernels solved a joint row on
one lane and walked a world's list on one thread; those rows had been compared
with the compiled reference, state by state.
"""
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(1, os.path.dirname(os.path.dirname(HERE)))
sys.path.append(os.path.dirname(os.path.dirname(os.path.dirname(HERE))))

import rbps_b200  # noqa: E402
from test_joint_states_gpu import SOLVES, states  # noqa: E402

if __name__ == "__main__":
    print(rbps_b200.LIB_PATH)
    out = {"%s %s" % (name, k): v for name, solve in SOLVES.items() for k, v in states(rbps_b200, solve).items()}
    np.savez_compressed(sys.argv[1] if len(sys.argv) > 1 else os.path.join(HERE, "states.npz"), **out)
