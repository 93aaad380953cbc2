"""The pool of page-locked readback blocks (rbps_b200/csrc/staging.hpp) on a
fake device: a block outlives its batch but not its context."""
import os
import subprocess

from conftest import ROOT


def test_staging_pool(tmp_path):
    exe = str(tmp_path / "staging")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", "-fsanitize=address,undefined",
                    "-I" + os.path.join(ROOT, "rbps_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "test_staging.cpp"), "-o", exe], check=True)
    # blocks that a reset leaves behind are dropped, not freed: no leak check
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120, env=dict(os.environ, ASAN_OPTIONS="detect_leaks=0"))
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
