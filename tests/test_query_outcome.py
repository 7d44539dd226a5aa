"""A query whose device wait gave up is reported as that, whatever its unwritten result words hold, in the
blocking form and by ticket: the outcome is taken from the status first (checked on the CPU, where the
timeout bit is simply set), and both callers take it from there."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "graphzeppelin_b200", "csrc")


def test_query_outcome(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "query_outcome_test")
    subprocess.run([gxx, "-std=c++14", "-O1", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpp", "query_outcome_test.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and "query outcome ok" in out.stdout, out.stdout


@pytest.mark.parametrize("function", ["int run_boruvka(", "int gz_query_wait("])
def test_results_are_read_after_the_outcome(function):
    """Neither caller returns rounds, labels or the component count before it has the outcome."""
    src = open(os.path.join(CSRC, "gz_capi.cu")).read()
    body = src[src.index(function):]
    body = body[:body.index("\n}\n")]
    at = body.index("query_outcome(")
    gave_up = body.index("QueryOutcome::kTimeout")
    assert at < gave_up
    for use in (r"\*rounds = ", r"last_rounds = ", r"last_ncc = ", r"\*num_cc = ", r"std::copy\(t.labels",
                r"boruvka_account\("):
        assert all(m.start() > gave_up for m in re.finditer(use, body)), use
