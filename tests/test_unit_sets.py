"""The sets in which a batch's situations run on the row chains, also after there was no memory for
larger ones: never more sets than task-counter slots (``tests/native/unit_sets_check.cpp``)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_sets_never_outnumber_the_counter_slots(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "unit_sets_check")
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "gral_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "unit_sets_check.cpp")], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=False).stdout.strip() == "ok"
