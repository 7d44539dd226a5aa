"""gz_spanning_forest moves the edges it returns and no more: a call for the count copies a few words, a
fetch 8 bytes an edge, whatever query form left the forest. Edge sets equal across the forms."""
import ctypes
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _handle(gz, V, mode, comps):
    from graphzeppelin_b200 import streams as S
    rng = np.random.default_rng(V)
    u = rng.integers(0, V, 3 * V)
    v = (u + comps * rng.integers(1, max(2, V // comps), 3 * V)) % (V - V % comps)  # same class mod comps
    keep = (u < V - V % comps) & (u != v)
    a = gz.CCSketchAlg(V, 6)
    a.set_query_graph(mode)
    a.ingest_records(S.make_records(u[keep].astype(np.uint32), v[keep].astype(np.uint32)))
    return a


def _copied(torch, tmp_path, f):
    """Bytes copied from the device to the host while f runs."""
    path = str(tmp_path / "trace.json")
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    p.export_chrome_trace(path)
    ev = [e for e in json.load(open(path))["traceEvents"] if "DtoH" in e.get("name", "")]
    assert ev  # the status words at least
    return sum(e["args"]["bytes"] for e in ev)


@pytest.mark.parametrize("V", [2, 1024, 1025, 40000])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_forest_has_its_edges_once(gz, V, mode):
    a = _handle(gz, V, mode, 1 if V == 2 else 7)
    n = ctypes.c_size_t()
    ncc = a.num_connected_components()
    assert a.lib.gz_spanning_forest(a._h, None, 0, ctypes.byref(n)) == 0 and n.value == V - ncc
    labels = a.connected_components().parent_arr
    for cap in (0, 1, V // 3, n.value, V):
        buf = np.full((V + 1, 2), 0xffffffff, np.uint32)
        assert a.lib.gz_spanning_forest(a._h, buf.ctypes.data, cap, ctypes.byref(n)) == 0
        got = min(cap, V - ncc)
        assert n.value == V - ncc and (buf[got:] == 0xffffffff).all()
        e = buf[:got].astype(np.int64)
        assert (e[:, 0] < e[:, 1]).all() and (e[:, 1] < V).all() and len({tuple(x) for x in e}) == got
        assert (labels[e[:, 0]] == labels[e[:, 1]]).all()
    a.close()


def test_forest_of_an_empty_graph(gz):
    with gz.CCSketchAlg(100, 1) as a:
        assert len(a.calc_spanning_forest().get_edges()) == 0


def test_forest_bytes(gz, tmp_path):
    torch = pytest.importorskip("torch")
    V = 200000
    a = _handle(gz, V, 2, 5)
    n = ctypes.c_size_t()
    want = V - a.num_connected_components()
    a.calc_spanning_forest()
    assert _copied(torch, tmp_path, lambda: a.lib.gz_spanning_forest(a._h, None, 0, ctypes.byref(n))) <= 64
    buf = np.empty((V, 2), np.uint32)
    assert _copied(torch, tmp_path, lambda: a.lib.gz_spanning_forest(
        a._h, buf.ctypes.data, want // 4, ctypes.byref(n))) <= 8 * (want // 4) + 64
    a.close()


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_forest_takes_no_memory_and_queries_go_on(gz, mode):
    """A fetch uses what the query left behind; later queries, traced or not, are as on a fresh handle."""
    torch = pytest.importorskip("torch")
    from graphzeppelin_b200 import streams as S
    V = 1 << 18
    a = _handle(gz, V, mode, 3)
    a.num_connected_components()
    rng = np.random.default_rng(3)
    more = S.make_records(rng.integers(0, V, 9).astype(np.uint32), rng.integers(0, V, 9).astype(np.uint32))
    before = torch.cuda.mem_get_info()[0]
    a.calc_spanning_forest()
    assert before - torch.cuda.mem_get_info()[0] < 1 << 20
    b = _handle(gz, V, mode, 3)
    for alg in (a, b):
        alg.set_trace(True)
        alg.ingest_records(more)
    x, y = a.connected_components(), b.connected_components()
    assert (x.parent_arr == y.parent_arr).all() and a.last_query_rounds == b.last_query_rounds
    assert sorted(a.get_trace().tolist()) == sorted(b.get_trace().tolist())
    assert len(a.calc_spanning_forest().get_edges()) == V - x.size()
    a.close()
    b.close()
