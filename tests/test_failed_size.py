"""A batch whose optional buffers (coded entries, the one-launch query's accumulators) do not fit asks for
them once, not in every call."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "graphzeppelin_b200", "csrc")


def test_failed_size(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "failed_size_test")
    subprocess.run([gxx, "-std=c++14", "-O1", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpp", "failed_size_test.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and "failed size ok" in out.stdout


@pytest.mark.parametrize("buffer,memo", [("grow(&h->d_entries, h->entry_cap, 4 * n_dense", "no_coded"),
                                         ("bool one_launch_buffers(gz_batch *h) {", "no_launch")])
def test_optional_buffers_ask_first(buffer, memo):
    src = open(os.path.join(CSRC, "gz_batch.cu")).read()
    at = src.index(buffer)
    near = src[at - 300:at + 1800]
    assert memo + ".may_try(" in near and memo + ".failed(" in near
