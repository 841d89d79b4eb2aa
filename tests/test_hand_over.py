"""The host's wait for the scalars that a launch writes to pinned memory, on the
CPU (tests/host/hand_over_check.cpp): words that come late, in any order or as the
writer's last act are taken; one that never comes is reported instead of being
taken for a value."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_words_late_missing_and_in_any_order(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "hand_over_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-pthread", os.path.join(ROOT, "tests", "host", "hand_over_check.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
