"""The on-chip CG's shapes (bounce_b200/csrc/resident_shape.h), checked on the
CPU: whatever numbering a cloth has, every row that a CTA's products read has a
thread that writes it.  The check is a small C++ program
(resident_shape_check.cpp) compiled with g++."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_every_halo_row_has_a_thread(tmp_path):
    exe = tmp_path / "resident_shape_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(exe), os.path.join(HERE, "resident_shape_check.cpp")],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip().endswith("ok")
