"""Which record calls go straight to the sketches is judged over everything that arrives between two
flushes, not call by call: a long stream in moderate calls fills the gutter and is applied as a wave."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_direct_route_properties(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "direct_route_test")
    subprocess.run([gxx, "-std=c++14", "-O1", "-Wall", "-Werror",
                    "-I", os.path.join(ROOT, "graphzeppelin_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "direct_route_test.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "direct route ok" in out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("V,n,calls", [(50021, 40000, 12), (1 << 17, 60000, 10)])
def test_stream_of_moderate_calls_fills_the_gutter(gz, V, n, calls):
    """Each call alone is below the direct threshold; together they are several times above it."""
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(V)
    rec = S.make_records(rng.integers(0, V, n * calls).astype(np.uint32),
                         rng.integers(0, V, n * calls).astype(np.uint32))
    with gz.CCSketchAlg(V, 3) as a, gz.CCSketchAlg(V, 3) as whole:
        for _ in range(2):  # a flush starts a new interval
            a.set_profiling(True)
            for i in range(calls):
                a.ingest_records(rec[i * n:(i + 1) * n])
            a.flush()
            p = a.get_profile()
            assert p["entries_applied"] == 2 * n * calls
            direct = calls - p["gutter_launches"]
            # at most 4 entries a vertex go direct, and one wave folds the rest
            assert 1 <= direct and direct * n < 2 * V and p["sketch_update_launches"] == direct + 1
        whole.ingest_records(rec)
        whole.ingest_records(rec)
        assert a.dump_sketches().tobytes() == whole.dump_sketches().tobytes()
