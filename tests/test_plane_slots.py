"""The plane kernel's partial sums (plane_steps.hpp, compiled for the host): no phase overwrites a
slot that other CTAs may still be reading, whatever order the phases come in."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_phase_writes_a_slot_that_is_still_read(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("needs g++")
    exe = str(tmp_path / "slots")
    subprocess.run(["g++", "-std=c++17", "-Wall", os.path.join(HERE, "cpp", "test_plane_slots.cpp"),
                    "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
