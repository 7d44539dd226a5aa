"""What the plane updates bring to L2 ahead of time lies inside the sketches, down to 2 vertices (one bucket a
column, where a fixed 64 bytes past the column's start would be 40 bytes past the last sketch)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "graphzeppelin_b200", "csrc")


def test_prefetches_stay_in_the_sketch(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "plane_layout_test")
    subprocess.run([gxx, "-std=c++14", "-O1", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpp", "plane_layout_test.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and "plane layout ok" in out.stdout


@pytest.mark.parametrize("file", ["gz_planes.cu", "gz_batch.cu"])
def test_no_fixed_distance(file):
    src = open(os.path.join(CSRC, file)).read()
    assert "column_second_word(" in src
    for line in src.splitlines():
        if "prefetch.global" in line:
            assert "+ 16)" not in line
